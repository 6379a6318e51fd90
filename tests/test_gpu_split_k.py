"""The fp16 product with its k split over a cluster, forced, where the sum of the partial tiles can go wrong:
fewer rows than CTAs, the rows of two tiles, columns that end inside a piece of four, unaligned and strided
outputs, each kind of store.

Tolerance: products of fp16 values are exact in fp32, and both sides add k of them in fp32 in their own order
(k * 2^-24 * sum |a b|); one rounding to fp16 of the sum and one of each operation of the store."""
import pytest
import torch

from adrastea_b200 import MatmulMask, MatmulOptions, MatmulStore, TensorLayout, TensorView

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [2, 4, 8])
@pytest.mark.parametrize("m,n,k,bn,pitch,step", [(1, 64, 1024, 64, 64, 1), (3, 131, 1032, 128, 131, 1), (64, 256, 1088, 256, 264, 1),
                                                 (130, 70, 2048, 64, 72, 1), (128, 40, 1024, 32, 82, 2), (200, 300, 1536, 128, 301, 1)])
@pytest.mark.parametrize("store,causal", [("identity", False), ("scale", True), ("add", False), ("bias", False)])
def test_split_k(kernels, split, m, n, k, bn, pitch, step, store, causal):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    half = lambda *s: torch.randn(s, device="cuda", generator=g).half()
    x, w, out0, bias = half(m, k), half(n, k), half(m, n), half(n)
    buf = torch.full((m * pitch + 8,), 5.0, dtype=torch.float16, device="cuda")
    out = torch.as_strided(buf, (m, n), (pitch, step))
    out.copy_(out0)
    opt = {"identity": MatmulStore.Identity(), "scale": MatmulStore.Scale(0.125), "add": MatmulStore.Add(),
           "bias": MatmulStore.BetaBias(0.5, TensorView.of(bias))}[store]
    kernels.set_tunable("tc_bn", bn)
    kernels.set_tunable("tc_split", split)
    try:
        kernels.matmul_f16(TensorView(buf, TensorLayout.new((m, n), (pitch, step))), TensorView.of(x),
                           TensorView.of(w).permute([1, 0]),
                           MatmulOptions.new().store(opt).mask(MatmulMask.Causal if causal else MatmulMask.None_))
    finally:
        kernels.set_tunable("tc_bn", 0)
        kernels.set_tunable("tc_split", 0)
    assert kernels.last_f16_schedule() == (bn, split, False)
    torch.cuda.synchronize()
    kernels.device_status()
    h = (x.float() @ w.float().t()).half().float()
    bound = (x.float().abs() @ w.float().abs().t()) * (k * 2.0 ** -24)
    want = {"identity": h, "scale": h * 0.125, "add": h + out0.float(),
            "bias": h + bias.float() + 0.5 * out0.float()}[store]
    tol = 2 * bound + 2.0 ** -10 * (h.abs() + want.abs() + bias.float().abs() + out0.float().abs()) + 2.0 ** -24
    got = out.float()
    if causal:
        hide = torch.triu(torch.ones(m, n, dtype=torch.bool, device="cuda"), 1)
        assert torch.isneginf(got[hide]).all()
        want, got = want.masked_fill(hide, 0.0), got.masked_fill(hide, 0.0)
    assert ((got - want).abs() <= tol).all()
    around = torch.ones_like(buf, dtype=torch.bool)
    torch.as_strided(around, (m, n), (pitch, step)).fill_(False)
    assert (buf[around] == 5.0).all()
