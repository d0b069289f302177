"""TTT-MLP backward kernel against float64 autograd over the CPU restatement of the reference's inner model."""

import pytest
import torch

from conftest import assert_close
from oracle import ttt_oracle as O

MLP_IN = ("xq", "xk", "xv", "w1", "b1", "w2", "b2", "token_eta", "ttt_lr_eta", "ln_weight", "ln_bias")


def _case(B, H, T, seed):
    t = O.make_inputs(B, H, T, 64, 16, seed=seed, dtype=torch.bfloat16, inner="mlp")
    g = torch.Generator().manual_seed(seed + 1)
    t["ln_weight"] = (1 + 0.1 * torch.randn(H, 64, generator=g)).to(torch.bfloat16)
    t["ln_bias"] = (0.1 * torch.randn(H, 64, generator=g)).to(torch.bfloat16)
    t["b1"] = (0.05 * torch.randn(B, H, 256, generator=g)).to(torch.bfloat16)
    t["b2"] = (0.05 * torch.randn(B, H, 64, generator=g)).to(torch.bfloat16)
    return t


@pytest.mark.gpu
@pytest.mark.parametrize("from_forward", (False, True))
@pytest.mark.parametrize("B,H,NS", ((1, 1, 1), (2, 3, 4), (1, 2, 12), (1, 1, 19)))
def test_mlp_backward_matches_autograd_of_the_restatement(B, H, NS, from_forward):
    """Both ways into the backward: on its own (it re-walks the sequence first), and on the workspace that the
    forward call filled on the way (final state + the operands of every state update)."""
    import ttt_rs_b200 as tb
    dev = torch.device("cuda:0")
    t = _case(B, H, NS * 16, 50 + NS)
    cfg = tb.FusedTttConfig.new(16, 64, 1e-6, 128, 1)
    d = {k: v.to(dev) for k, v in t.items()}
    st = tb.TTTMLPState(d["w1"], d["b1"], d["w2"], d["b2"])
    ws = None
    if from_forward:
        ws = tb.mlp_backward_workspace(d["xq"], cfg)
        tb.fused_ttt_mlp_forward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                                 d["ln_bias"], cfg, backward_workspace=ws)
    g = tb.fused_ttt_mlp_backward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                                  d["ln_bias"], d["grad_output"], cfg, workspace_from_forward=ws)
    torch.cuda.synchronize()
    tb.check_mlp_status(g)
    want = O.ttt_mlp_backward_autograd(*[t[k].double() for k in MLP_IN], t["grad_output"].double())
    fold = lambda x: x.double().cpu().reshape(-1, 16).sum(0)  # noqa: E731  token_eta gradient per position
    for k in ("grad_xq", "grad_xk", "grad_xv", "grad_w1", "grad_b1", "grad_w2", "grad_b2", "grad_ttt_lr_eta",
              "grad_ln_weight", "grad_ln_bias"):
        assert_close(g[k], want[k], 2e-2, k, max_bad_frac=1e-3)  # twice the worst fraction measured on B200 (4.9e-4)
    # token_eta: every (stage, position) entry at the bf16 tolerance.  The sum over the stages of one position can
    # cancel heavily (entries of both signs; for position 15, which also carries the step-size gradient of the state
    # updates, |sum| is up to 30 times smaller than the sum of the magnitudes), so the folded vector is held to the
    # usual criterion or to 5e-3 of the sum of the magnitudes of its terms, whichever is larger.
    assert_close(g["grad_token_eta"], want["grad_token_eta"], 2e-2, "grad_token_eta (per stage and position)")
    fw = fold(want["grad_token_eta"])
    err = (fold(g["grad_token_eta"]) - fw).abs()
    bound = torch.maximum(2e-2 * (fw.abs() + fw.pow(2).mean().sqrt()), 5e-3 * fold(want["grad_token_eta"].abs()))
    assert bool((err <= bound).all()), f"grad_token_eta folded: error {err.tolist()} above {bound.tolist()}"


@pytest.mark.gpu
def test_mlp_backward_at_the_benchmark_size_on_sampled_streams():
    """Config 2 in full (B=16 H=12 T=2048: 192 streams on 148 persistent blocks, 128 stages); the streams are
    independent, so three of them are checked against float64 autograd and the batch reductions by linearity."""
    import ttt_rs_b200 as tb
    dev = torch.device("cuda:0")
    B, H, T = 16, 12, 2048
    t = O.make_inputs(B, H, T, 64, 16, seed=0, dtype=torch.bfloat16, inner="mlp")
    cfg = tb.FusedTttConfig.new(16, 64, 1e-6, 128, 1)
    d = {k: v.to(dev) for k, v in t.items()}
    st = tb.TTTMLPState(d["w1"], d["b1"], d["w2"], d["b2"])
    ws = tb.mlp_backward_workspace(d["xq"], cfg)
    tb.fused_ttt_mlp_forward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                             d["ln_bias"], cfg, backward_workspace=ws)
    g = tb.fused_ttt_mlp_backward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                                  d["ln_bias"], d["grad_output"], cfg, workspace_from_forward=ws)
    torch.cuda.synchronize()
    tb.check_mlp_status(g)  # 192 streams x 16 work items handed between the persistent blocks, no wait ran out
    for k, v in g.items():
        if not k.startswith("_"):
            assert torch.isfinite(v.float()).all(), k
    for b, h in ((0, 0), (7, 5), (15, 11)):  # first wave, middle, last stream of the second wave
        one = {k: (v[b:b + 1, h:h + 1] if v.dim() >= 3 else v) for k, v in t.items()}
        one["ln_weight"], one["ln_bias"] = t["ln_weight"][h:h + 1], t["ln_bias"][h:h + 1]
        want = O.ttt_mlp_backward_autograd(*[one[k].double() for k in MLP_IN], one["grad_output"].double())
        for k in ("grad_xq", "grad_xk", "grad_xv", "grad_w1", "grad_b1", "grad_w2", "grad_b2", "grad_ttt_lr_eta"):
            assert_close(g[k][b:b + 1, h:h + 1], want[k], 2e-2, f"stream ({b},{h}) {k}", max_bad_frac=1e-3)  # measured at most 4.9e-4
    # a second run gives the same bits (fixed-order reductions, no atomics)
    tb.fused_ttt_mlp_forward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                             d["ln_bias"], cfg, backward_workspace=ws)
    g2 = tb.fused_ttt_mlp_backward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                                   d["ln_bias"], d["grad_output"], cfg, workspace_from_forward=ws)
    torch.cuda.synchronize()
    for k in ("grad_xq", "grad_w1", "grad_token_eta", "grad_ln_weight"):
        assert torch.equal(g[k], g2[k]), f"{k} differs between two runs"
    # and the backward that walks the sequence itself (32 work items per stream) agrees with it
    g3 = tb.fused_ttt_mlp_backward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                                   d["ln_bias"], d["grad_output"], cfg)
    torch.cuda.synchronize()
    tb.check_mlp_status(g3)
    for k in ("grad_xq", "grad_xk", "grad_w1", "grad_w2", "grad_ttt_lr_eta"):
        assert_close(g3[k], g[k].float(), 2e-2, f"{k}: own forward walk vs workspace from the forward",
                     max_bad_frac=2.5e-4)  # measured at most 1.1e-4


@pytest.mark.gpu
def test_mlp_autograd_node():
    """`fused_ttt_mlp` under torch autograd: gradients reach the leaves and equal the direct calls (forward filling
    the backward's workspace, then the backward on it)."""
    import ttt_rs_b200 as tb
    dev = torch.device("cuda:0")
    t = _case(1, 2, 32, 77)
    cfg = tb.FusedTttConfig.new(16, 64, 1e-6, 128, 1)
    d = {k: v.to(dev) for k, v in t.items()}
    leaves = {k: d[k].clone().requires_grad_(True) for k in ("xq", "xk", "xv", "w1", "b1", "w2", "b2", "ttt_lr_eta",
                                                             "ln_weight", "ln_bias")}
    out, _ = tb.fused_ttt_mlp(leaves["xq"], leaves["xk"], leaves["xv"],
                              tb.TTTMLPState(leaves["w1"], leaves["b1"], leaves["w2"], leaves["b2"]), d["token_eta"],
                              leaves["ttt_lr_eta"], leaves["ln_weight"], leaves["ln_bias"], cfg)
    out.backward(d["grad_output"])
    st = tb.TTTMLPState(d["w1"], d["b1"], d["w2"], d["b2"])
    ws = tb.mlp_backward_workspace(d["xq"], cfg)
    tb.fused_ttt_mlp_forward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                             d["ln_bias"], cfg, backward_workspace=ws)
    g = tb.fused_ttt_mlp_backward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                                  d["ln_bias"], d["grad_output"], cfg, workspace_from_forward=ws)
    torch.cuda.synchronize()
    for k in ("xq", "xk", "xv", "w1", "b1", "w2", "b2", "ttt_lr_eta"):
        assert torch.equal(leaves[k].grad, g["grad_" + k]), k
    assert torch.equal(leaves["ln_weight"].grad, g["grad_ln_weight"].to(torch.bfloat16))


@pytest.mark.gpu
@pytest.mark.parametrize("from_forward", (False, True))
def test_mlp_backward_is_bitwise_reproducible(from_forward):
    """More streams than persistent blocks (B=16 H=12: 192 streams, 4 work items each), so a stream's items run on
    different SMs and its float32 state travels tensor memory -> workspace -> tensor memory between them; a dirty
    workspace the second time round.  Any race in those hand-offs, or a read of tensor memory or of the bf16 operand
    copies that the run did not write itself, shows up as a difference between two runs."""
    import ttt_rs_b200 as tb
    dev = torch.device("cuda:0")
    B, H, T = 16, 12, 512
    t = O.make_inputs(B, H, T, 64, 16, seed=3, dtype=torch.bfloat16, inner="mlp")
    cfg = tb.FusedTttConfig.new(16, 64, 1e-6, 128, 1)
    d = {k: v.to(dev) for k, v in t.items()}
    st = tb.TTTMLPState(d["w1"], d["b1"], d["w2"], d["b2"])
    ws = tb.mlp_backward_workspace(d["xq"], cfg) if from_forward else None
    runs = []
    for _ in range(2):
        if from_forward:
            tb.fused_ttt_mlp_forward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                                     d["ln_bias"], cfg, backward_workspace=ws)
        g = tb.fused_ttt_mlp_backward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                                      d["ln_bias"], d["grad_output"], cfg, workspace_from_forward=ws)
        torch.cuda.synchronize()
        tb.check_mlp_status(g)
        runs.append({k: v.clone() for k, v in g.items() if k.startswith("grad_")})  # (not the scratch it carries along)
    assert len(runs[0]) == 11
    for k in runs[0]:
        assert torch.equal(runs[0][k], runs[1][k]), f"{k} differs between two runs"
    assert all(bool(torch.isfinite(v.float()).all()) for v in runs[0].values())


@pytest.mark.gpu
def test_rows_off_their_centre():
    """Z2 and Zb2 rows whose mean is about 100 times their standard deviation: the gradients differentiate both LayerNorms with
    variances summed about the mean.  From E[z^2] - mean^2 in float32 the variance would be off by up to 100^2 2^-22 = 2.4e-3,
    a bias of every row (grad_w1 of this case: 1.1e-2 off in 2-norm, against 3.7e-3).  The other errors are those of centred
    rows, bf16 operands (largest here: 4.3e-3), plus 2.4e-3 through the forward's own inner gradients: 7e-3 holds both."""
    import ttt_rs_b200 as tb
    dev = torch.device("cuda:0")
    t = _case(1, 8, 256, 5)
    g = torch.Generator().manual_seed(6)
    t["b2"] = (2.0 + 0.01 * torch.randn(1, 8, 64, generator=g)).to(torch.bfloat16)
    cfg = tb.FusedTttConfig.new(16, 64, 1e-6, 128, 1)
    d = {k: v.to(dev) for k, v in t.items()}
    want = O.ttt_mlp_backward_autograd(*[d[k].double() for k in MLP_IN], d["grad_output"].double())
    st = tb.TTTMLPState(d["w1"], d["b1"], d["w2"], d["b2"])
    got = tb.fused_ttt_mlp_backward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                                    d["ln_bias"], d["grad_output"], cfg)
    torch.cuda.synchronize()
    tb.check_mlp_status(got)
    for k in ("grad_xq", "grad_xk", "grad_xv", "grad_w1", "grad_b1", "grad_w2", "grad_b2", "grad_ttt_lr_eta",
              "grad_ln_weight", "grad_ln_bias"):
        err = ((got[k].double() - want[k]).norm() / want[k].norm()).item()
        print(f"{k}: {err:.2e}")
        assert err < 7e-3, f"{k}: {err}"


@pytest.mark.gpu
@pytest.mark.parametrize("from_forward", (False, True))
@pytest.mark.parametrize("B,H,NS,te_scale,bound", ((1, 3, 9, 0.0, 1e-2), (1, 3, 24, 0.7, 1e-2), (1, 4, 512, 1.0, 2e-2)))
def test_step_scales_and_many_stages(B, H, NS, te_scale, bound, from_forward):
    """The masters of W1, W2 are carried divided by -token_eta[15] and undone stage by stage: token_eta[15] = 0 (nothing moves and
    nothing is undone), a token_eta[15] that is no power of two (bf16(0.7 / 16): the division rounds), and 512 stages.
    bf16 operands give gradients 2e-3 to 4e-3 off (2-norm; 1e-2 is the bf16 tolerance of these tests' L2 errors); over 512 stages
    the state's own rounding comes back through the chain, up to 1e-2 (grad_b1).  Where the undone state has drifted longest, in
    the first four stages, the gradients of the tokens are held to the bound of a short sequence."""
    import ttt_rs_b200 as tb
    dev = torch.device("cuda:0")
    t = _case(B, H, NS * 16, 200 + NS)
    te = t["token_eta"].float().view(-1, 16)
    if te_scale == 0.0:
        te[:, 15] = 0.0
    else:
        te = te * te_scale
    t["token_eta"] = te.reshape(-1).to(torch.bfloat16)
    cfg = tb.FusedTttConfig.new(16, 64, 1e-6, 128, 1)
    d = {k: v.to(dev) for k, v in t.items()}
    st = tb.TTTMLPState(d["w1"], d["b1"], d["w2"], d["b2"])
    ws = None
    if from_forward:
        ws = tb.mlp_backward_workspace(d["xq"], cfg)
        tb.fused_ttt_mlp_forward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                                 d["ln_bias"], cfg, backward_workspace=ws)
    g = tb.fused_ttt_mlp_backward(d["xq"], d["xk"], d["xv"], st, d["token_eta"], d["ttt_lr_eta"], d["ln_weight"],
                                  d["ln_bias"], d["grad_output"], cfg, workspace_from_forward=ws)
    torch.cuda.synchronize()
    tb.check_mlp_status(g)
    want = O.ttt_mlp_backward_autograd(*[d[k].double() for k in MLP_IN], d["grad_output"].double())
    for k in ("grad_xq", "grad_xk", "grad_xv", "grad_w1", "grad_b1", "grad_w2", "grad_b2", "grad_ttt_lr_eta",
              "grad_ln_weight", "grad_ln_bias"):
        err = ((g[k].double() - want[k]).norm() / want[k].norm()).item()
        print(f"{k}: {err:.2e}")
        assert err < bound, f"{k}: {err}"
    for k in ("grad_xq", "grad_xk", "grad_xv"):
        a, b = g[k][:, :, :64].double(), want[k][:, :, :64]
        err = ((a - b).norm() / b.norm()).item()
        print(f"{k}, first stages: {err:.2e}")
        assert err < 1e-2, f"{k}, first stages: {err}"


@pytest.mark.gpu
@pytest.mark.parametrize("offset", (1, 4))
def test_walk_takes_a_second_layer_at_any_address(offset):
    """w2 sliced out of a flat buffer, 2 or 8 bytes past a 16-byte boundary: the same gradients, bit for bit."""
    import ttt_rs_b200 as tb
    dev = torch.device("cuda:0")
    t = _case(1, 3, 48, 91)
    cfg = tb.FusedTttConfig.new(16, 64, 1e-6, 128, 1)
    d = {k: v.to(dev) for k, v in t.items()}
    flat = torch.zeros(d["w2"].numel() + 8, dtype=torch.bfloat16, device=dev)
    sliced = flat[offset:offset + d["w2"].numel()].view_as(d["w2"])
    sliced.copy_(d["w2"])
    assert sliced.data_ptr() % 16 == 2 * offset
    got = []
    for w2 in (d["w2"], sliced):
        g = tb.fused_ttt_mlp_backward(d["xq"], d["xk"], d["xv"], tb.TTTMLPState(d["w1"], d["b1"], w2, d["b2"]), d["token_eta"],
                                      d["ttt_lr_eta"], d["ln_weight"], d["ln_bias"], d["grad_output"], cfg)
        torch.cuda.synchronize()
        tb.check_mlp_status(g)
        got.append(g)
    for k in got[0]:
        if k.startswith("grad_"):
            assert torch.equal(got[0][k], got[1][k]), k
