"""The layer's epilogue (post LayerNorm, optional gate) against plain PyTorch in float32, at the edges of the kernel's tiling:
token counts that do not fill a tile, rows of one head, the widest row of each instantiation and the narrowest of the next."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gate", [False, True])
@pytest.mark.parametrize("dtype,B,H,T,F", [
    (torch.bfloat16, 1, 1, 1, 64), (torch.bfloat16, 3, 5, 37, 64), (torch.bfloat16, 2, 16, 17, 64),
    (torch.bfloat16, 2, 17, 15, 64), (torch.bfloat16, 1, 32, 9, 64), (torch.bfloat16, 2, 2, 33, 32),
    (torch.float32, 1, 1, 1, 64), (torch.float32, 2, 8, 19, 64), (torch.float32, 2, 9, 7, 64),
    (torch.float32, 1, 17, 5, 64), (torch.float32, 1, 32, 3, 64), (torch.float32, 2, 6, 21, 32)])
def test_epilogue(dtype, B, H, T, F, gate):
    from ttt_rs_b200 import layer as L
    gen = torch.Generator(device="cuda").manual_seed(H * 100 + T)
    C = H * F
    mk = lambda *s: torch.randn(*s, device="cuda", generator=gen).to(dtype)  # noqa: E731
    x, w, b = mk(B, H, T, F), mk(C), mk(C)
    g = mk(B * T, C + 4) if gate else None  # a pitch that leaves rows aligned to 8 (16) bytes only
    y = L.layer_epilogue(x, w, b, 1e-6, g, C + 4 if gate else 0)
    want = torch.nn.functional.layer_norm(x.float().transpose(1, 2).reshape(B, T, C), (C,), w.float(), b.float(), 1e-6)
    if gate:
        want = want * torch.nn.functional.gelu(g[:, :C].float(), approximate="tanh").reshape(B, T, C)
    tol = 1e-2 if dtype == torch.bfloat16 else 1e-5
    assert (y.float() - want).norm() <= tol * want.norm()


@pytest.mark.parametrize("gate", [False, True])
@pytest.mark.parametrize("dtype,H,F", [
    (torch.bfloat16, 1, 32), (torch.bfloat16, 4, 32), (torch.bfloat16, 5, 32), (torch.bfloat16, 7, 64), (torch.bfloat16, 18, 32),
    (torch.bfloat16, 19, 32), (torch.bfloat16, 23, 32), (torch.bfloat16, 24, 32), (torch.float32, 7, 64), (torch.float32, 13, 64)])
def test_tile_rules(dtype, H, F, gate):
    """The widths on both sides of each line of the rule for groups, rows and threads, on a tile and a ragged rest."""
    test_epilogue(dtype, 2, H, 29, F, gate)
