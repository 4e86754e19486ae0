"""The grouped GEMM of the gated experts against 64-bit products per expert."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,K,cols", [
    ([0, 1, 31, 32, 33, 0, 255, 256, 257, 300, 0], 72, 40),          # tails of K, of the columns, of the tokens; empty experts at both ends
    ([5, 700, 64, 1025], 512, 264), ([1] * 8, 64, 8), ([3, 0, 520], 1000, 1024),
    ([1, 0, 2] * 700, 64, 16),                                       # more experts than one launch takes
])
@pytest.mark.parametrize("glu,weights", [(None, False), ((float("inf"), 1.0, 0.0), True), ((7.0, 1.702, 1.0), False)])
def test_grouped_gemm_matches_64_bit_products(cuda_device, rows, K, cols, glu, weights):
    """fp32 sums of exact products and the activation are off by a few 1e-6, far below the 2e-5 allowed here;
    the output rounds to bf16 once: 2^-8 of it at most."""
    from jax_gpt_b200 import _ext
    g = torch.Generator(device=cuda_device).manual_seed(5)
    E, R, d = len(rows), sum(rows), torch.float64
    rnd = lambda *s: torch.randn(*s, device=cuda_device, generator=g)
    xs = rnd(R, K).bfloat16()
    w = (rnd(E, cols * (2 if glu else 1), K + 8) * K ** -0.5).bfloat16()[..., :K]       # rows further apart than their length
    w_row = rnd(R).abs() if weights else None
    ends = torch.tensor(rows, device=cuda_device).cumsum(0).to(torch.int32)
    out = torch.full((R + 1, cols), 3.0, device=cuda_device, dtype=torch.bfloat16)
    _ext.ops().grouped_gemm(xs, w, ends, glu, w_row, out[:R])
    ref, at = torch.empty(R, cols, device=cuda_device, dtype=d), 0
    for e, n in enumerate(rows):
        if n:
            y = xs[at:at + n].to(d) @ w[e].to(d).t()
            if glu:
                y = y * (w_row[at:at + n, None].to(d) if weights else 1.0)
                gate, up = y[:, :cols].clamp(max=glu[0]), y[:, cols:].clamp(-glu[0], glu[0])
                y = gate * torch.sigmoid(glu[1] * gate) * (up + glu[2])
            ref[at:at + n] = y
        at += n
    err = (out[:R].to(d) - ref).abs()
    assert (err <= 2.0 ** -8 * ref.abs() * 1.001 + 2e-5).all(), (err - 2.0 ** -8 * ref.abs()).max().item()
    assert (out[R] == 3.0).all()
