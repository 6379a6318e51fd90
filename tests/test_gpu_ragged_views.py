"""fp16 products of views with odd pitches and unaligned bases: operands read in aligned 16-byte chunks
shifted together, outputs written through a staging tile.  The operands lie in buffers of NaN and the
output in a buffer of canaries, so an element taken from or written beside a view shows.

Tolerance: products of fp16 values are exact in fp32, and both sides add k of them in fp32 in their own
order (k * 2^-24 * sum |a b|); one rounding to fp16 of the sum and one of each operation of the store."""
import pytest
import torch

from adrastea_b200 import MatmulMask, MatmulOptions, MatmulStore, TensorLayout, TensorView

pytestmark = pytest.mark.gpu


def view(t, pitch, lead, fill):
    """t [b, r, c] inside a 1-D buffer: rows `pitch` apart, `lead` elements before the first."""
    b, r, c = t.shape
    buf = torch.full((lead + b * r * pitch + 24,), fill, dtype=torch.float16, device="cuda")
    inner = buf[lead:lead + b * r * pitch].view(b, r, pitch)[:, :, :c]
    inner.copy_(t)
    return buf, inner, TensorView(buf[lead:], TensorLayout.new((b, r, c), (r * pitch, pitch, 1)))


# pitches of every parity, bases at every offset in a 16-byte chunk, widths around a piece, a k-block and a
# tile, one element; rhs as rows of k and as rows of n
@pytest.mark.parametrize("kmajor", [False, True])
@pytest.mark.parametrize("b,m,n,k,gap,lead", [(2, 257, 64, 257, 0, 0), (3, 5, 9, 7, 1, 1), (1, 130, 129, 65, 2, 2),
                                              (2, 33, 31, 63, 3, 3), (1, 1, 1, 1, 0, 4), (2, 129, 257, 64, 5, 5),
                                              (1, 64, 40, 200, 6, 6), (2, 128, 300, 129, 7, 7)])
@pytest.mark.parametrize("store,causal", [("identity", False), ("scale", True), ("add", False), ("bias", False)])
def test_ragged_views(kernels, b, m, n, k, gap, lead, kmajor, store, causal):
    g = torch.Generator(device="cuda").manual_seed(m * 31 + n + k)
    half = lambda *s: torch.randn(s, device="cuda", generator=g).half()
    x, w, out0, bias = half(b, m, k), half(b, k, n), half(b, m, n), half(n)
    _, _, xv = view(x, k + gap, lead, float("nan"))
    if kmajor:
        _, _, wv = view(w.transpose(1, 2), k + gap, lead, float("nan"))
        wv = wv.permute([0, 2, 1])
    else:
        _, _, wv = view(w, n + gap, lead, float("nan"))
    buf, out, ov = view(out0, n + gap, lead, 5.0)
    opt = {"identity": MatmulStore.Identity(), "scale": MatmulStore.Scale(0.125), "add": MatmulStore.Add(),
           "bias": MatmulStore.BetaBias(0.5, TensorView.of(bias))}[store]
    kernels.matmul_f16(ov, xv, wv, MatmulOptions.new().store(opt).mask(MatmulMask.Causal if causal else MatmulMask.None_))
    torch.cuda.synchronize()
    kernels.device_status()
    h = (x.float() @ w.float()).half().float()
    bound = (x.float().abs() @ w.float().abs()) * (k * 2.0 ** -24)
    want = {"identity": h, "scale": h * 0.125, "add": h + out0.float(),
            "bias": h + bias.float() + 0.5 * out0.float()}[store]
    tol = 2 * bound + 2.0 ** -10 * (h.abs() + want.abs() + bias.float().abs() + out0.float().abs()) + 2.0 ** -24
    got = out.float()
    if causal:
        hide = torch.triu(torch.ones(m, n, dtype=torch.bool, device="cuda"), 1)
        assert torch.isneginf(got[:, hide]).all()
        want, got = want.masked_fill(hide, 0.0), got.masked_fill(hide, 0.0)
    assert ((got - want).abs() <= tol).all()
    around = torch.ones_like(buf, dtype=torch.bool)
    around[lead:lead + b * m * (n + gap)].view(b, m, n + gap)[:, :, :n] = False
    assert (buf[around] == 5.0).all()
