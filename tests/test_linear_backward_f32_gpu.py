"""The float32 TTT-Linear backward: a stream on an SM of its own, walked in one piece, and more streams than SMs, walked in
chunks that hand the state on, give the same bits; both match the oracle."""

import pytest
import torch

from conftest import assert_close
from oracle import ttt_oracle as O

IN = ("xq", "xk", "xv", "weight", "bias", "token_eta", "ttt_lr_eta", "ln_weight", "ln_bias")


@pytest.mark.gpu
@pytest.mark.parametrize("F,mb", ((64, 16), (32, 16), (64, 8), (32, 8)))
@pytest.mark.parametrize("NS,K", (
    (17, 16),  # a chunk of one stage; chunks end where checkpoints do
    (35, 5),   # chunks that end inside a checkpoint interval: W is handed on
    (33, 64),  # one checkpoint for the sequence
))
def test_chunks_equal_one_piece_and_the_oracle(F, mb, NS, K):
    import ttt_rs_b200 as tb
    dev = torch.device("cuda:0")
    H = 4 * (64 // F)
    B = 2 * (torch.cuda.get_device_properties(dev).multi_processor_count // 8 + 1)  # 4 B tiles > SMs >= 2 B
    t = O.make_inputs(B, H, NS * mb, F, mb, seed=NS + K, dtype=torch.float32)
    cfg = tb.FusedTttConfig.new(mb, F, 1e-6, 128, K)
    batched = [k for k in IN if t[k].shape[0] == B and t[k].dim() >= 3]

    def run(sel):
        ts = [(t[k][sel] if k in batched else t[k]).to(dev).contiguous().requires_grad_(True) for k in IN]
        tb.fused_ttt_tile_forward_multi(*ts, cfg)[0].backward(t["grad_output"][sel].to(dev).contiguous())
        tb.check_status()
        return {k: x.grad for k, x in zip(IN, ts)}

    whole, lo, hi = run(slice(0, B)), run(slice(0, B // 2)), run(slice(B // 2, B))
    one = slice(B - 1, B)  # (a stream that the last blocks take)
    ref = O.ttt_linear_backward(*[(t[k][one] if k in batched else t[k]).double() for k in IN], t["grad_output"][one].double(),
                                mini_batch=mb, eps=1e-6)
    for k in IN:
        if k in batched:
            assert torch.equal(whole[k], torch.cat([lo[k], hi[k]])), k
            assert_close(whole[k][one], ref["grad_" + k], 1e-4, "grad_" + k)
        else:  # sums over the streams, in an order of each launch's own: a few hundred additions of 2^-24 each
            a, b = whole[k].double(), lo[k].double() + hi[k].double()
            assert ((a - b).norm() / b.norm()).item() < 1e-5, k


@pytest.mark.gpu
def test_a_handoff_that_never_comes_ends_the_launch():
    """The first item numbers are skipped, so the chain group of every block waits for a hand-off that nothing publishes: its
    bounded wait ends the other groups' waits, the launch returns, and the next one gives the earlier gradients."""
    import ttt_rs_b200 as tb
    from ttt_rs_b200 import _lib
    dev = torch.device("cuda:0")
    B, H = 40, 4
    t = O.make_inputs(B, H, 32 * 16, 64, 16, seed=3, dtype=torch.float32)
    cfg = tb.FusedTttConfig.new(16, 64, 1e-6, 128, 16)
    outs, saved = tb.TttTileMultiKernel.forward_launch(tb.TttInputs(*[t[k].to(dev).contiguous() for k in IN]), cfg)
    go = tb.TttOutputs(t["grad_output"].to(dev), None, None)
    good = tb.TttTileMultiKernel.backward_launch(saved, go, cfg)
    tb.check_status()
    lib = _lib.load()
    try:
        lib.ttt_b200_debug_handoff(2000, B * H)
        bad = tb.TttTileMultiKernel.backward_launch(saved, go, cfg)
        torch.cuda.synchronize()
    finally:
        lib.ttt_b200_debug_handoff(0, 0)
    words = bad.status.cpu().tolist()
    assert words[0] == _lib.TTT_ERR_TIMEOUT and words[1] == 15 and words[3] == 15, words
    with pytest.raises(tb.TttError):
        tb.check_status()
    again = tb.TttTileMultiKernel.backward_launch(saved, go, cfg)
    tb.check_status()
    for n in IN:
        assert torch.equal(getattr(again, n), getattr(good, n)), n
