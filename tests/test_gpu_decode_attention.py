"""Decode attention in one pass over the cache, and the form that also rotates and appends the new token.

The fused form runs the same arithmetic on the same values as decode_rope_append followed by
decode_attention, so outputs and caches have the same bits.  Against fp32 attention over the cache: scores
are rounded to fp16 twice (relative 2^-10 of a score of at most `top` shifts a probability by at most
2 * 2^-10 * top relative), the output once (2^-11); fp32 sums add nothing that shows."""
import pytest
import torch

from adrastea_b200 import TensorView

pytestmark = pytest.mark.gpu


# every number of CTAs per (head, sequence); fewer positions than CTAs, lanes and steps; one past a step
# of all warps; the first and the last position of the cache; a position outside it; more CTAs than run at once
# with eight steps in flight, for each head size split four and eight ways; whole steps of cached positions with
# the new one behind them and as the last of them
@pytest.mark.parametrize("cs", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("B,H,hd,S,pos", [(1, 32, 128, 640, 575), (3, 5, 64, 136, 128), (2, 3, 256, 72, 64),
                                          (1, 1, 128, 8, 0), (2, 4, 128, 16, 15), (16, 32, 128, 80, 65),
                                          (1, 2, 64, 2048, 2047), (2, 2, 128, 16, 16), (1, 2, 256, 16, -1),
                                          (3, 32, 64, 136, 130), (1, 40, 64, 136, 130), (3, 32, 128, 72, 70),
                                          (1, 40, 128, 72, 70), (3, 32, 256, 40, 33), (1, 40, 256, 40, 33),
                                          (2, 2, 128, 264, 256), (2, 2, 128, 256, 255)])
def test_decode_rope_attention(kernels, cs, B, H, hd, S, pos):
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + hd + pos + 1)
    half = lambda *s: torch.randn(s, device="cuda", generator=g).half()
    width = H * hd
    qkv, kc, vc = half(B, 3 * width), half(B, S, width), half(B, S, width)
    at = torch.tensor([pos], dtype=torch.int32, device="cuda")
    scale = 1.0 / hd ** 0.5
    view = lambda t, i: TensorView.of(t[:, i * width:(i + 1) * width])
    kernels.set_tunable("att_cs", cs)
    try:
        one, k1, v1 = torch.full((B, width), 3.0, dtype=torch.float16, device="cuda"), kc.clone(), vc.clone()
        kernels.decode_rope_attention(TensorView.of(one), *(view(qkv, i) for i in range(3)), k1, v1, H, at,
                                      10000.0, scale)
        two, k2, v2, turned = torch.empty_like(one), kc.clone(), vc.clone(), qkv.clone()
        kernels.decode_rope_append(*(view(turned, i) for i in range(3)), k2, v2, H, at, 10000.0)
        kernels.decode_attention(TensorView.of(two), view(turned, 0), k2, v2, H, at, scale)
    finally:
        kernels.set_tunable("att_cs", 0)
    torch.cuda.synchronize()
    kernels.device_status()
    assert torch.equal(one, two) and torch.equal(k1, k2) and torch.equal(v1, v2)
    T = min(max(pos + 1, 0), S)
    if T == 0:
        assert not one.any()
        return
    heads = lambda t: t[:, :T].float().view(B, T, H, hd).permute(0, 2, 1, 3)
    q = turned[:, :width].float().view(B, H, 1, hd)
    s = (q @ heads(k2).transpose(-1, -2)) * scale
    want = (s.softmax(-1) @ heads(v2)).view(B, width)
    top = s.abs().max().item()
    tol = (2 * 2.0 ** -10 * top + 2.0 ** -11) * heads(v2).abs().amax().item()
    assert (one.float() - want).abs().max().item() <= tol
