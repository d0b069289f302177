"""The two forms of the TTT-Linear forward (streams that share SMs / streams with an SM each) give the same bits."""

import pytest
import torch

from oracle import ttt_oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("mb", (16, 8))
@pytest.mark.parametrize("F", (64, 32))
@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float32))
@pytest.mark.parametrize("NS", (1, 2, 5, 9))
def test_more_streams_than_sms_equal_their_halves(dtype, F, mb, NS):
    """All streams in one launch are more than the SMs, each half is fewer; NS around the depths of the two forms' rings.
    Both forms do the same operations in the same order, so everything per stream is equal bit for bit -- also what
    the backward makes of the saved state."""
    import ttt_rs_b200 as tb
    dev = torch.device("cuda:0")
    per_tile = 64 // F
    H = 4 * per_tile
    B = 2 * (torch.cuda.get_device_properties(dev).multi_processor_count // 8 + 1)  # 4 B streams > SMs >= 2 B
    t = O.make_inputs(B, H, NS * mb, F, mb, seed=NS, dtype=dtype)
    cfg = tb.FusedTttConfig.new(mb, F, 1e-6, 128, 4)
    names = ("xq", "xk", "xv", "weight", "bias", "token_eta", "ttt_lr_eta", "ln_weight", "ln_bias")
    batched = [k for k in names if t[k].shape[0] == B and t[k].dim() >= 3]

    def run(sel):
        ts = [(t[k][sel] if k in batched else t[k]).to(dev).contiguous().requires_grad_(True) for k in names]
        res = tb.fused_ttt_tile_forward_multi(*ts, cfg)
        res[0].backward(t["grad_output"][sel].to(dev).contiguous())
        return [r.detach() for r in res] + [x.grad for k, x in zip(names, ts) if k in batched]

    whole = run(slice(0, B))
    halves = [run(slice(0, B // 2)), run(slice(B // 2, B))]
    for i, w in enumerate(whole):
        assert torch.equal(w, torch.cat([h[i] for h in halves])), i
        assert bool(torch.isfinite(w.float()).all()), i
