"""The fp16 product on CTA pairs (256 x 256 tiles), forced on sizes around its tiles, against an fp32
product of the same fp16 operands.

Tolerance: products of fp16 values are exact in fp32 and both sides add k of them in fp32, so they
differ by the order of the additions, at most k * 2^-24 * sum |a b| (taken with sum |a b| from the
operands), plus one rounding to fp16 of the result and one of each fp16 operation of the store."""
import pytest
import torch

from adrastea_b200 import MatmulLoad, MatmulMask, MatmulOptions, MatmulStore, TensorLayout, TensorView

pytestmark = pytest.mark.gpu


def half(g, *shape):
    return torch.randn(shape, device="cuda", generator=g).half()


def expected(x, w, out0, bias, store, causal):
    acc = x.float() @ w.float()
    bound = (x.float().abs() @ w.float().abs()) * (x.shape[-1] * 2.0 ** -24)
    h = acc.half().float()
    b, o = bias.float(), out0.float()
    want = {"identity": h, "scale": h * 0.125, "add": h + o, "bias": h + b, "beta_bias": h + b + 0.5 * o,
            "quick_gelu": (h + b) * torch.sigmoid(1.702 * (h + b)),
            "beta_gelu": torch.nn.functional.gelu(h + b, approximate="tanh") + 0.5 * o}[store]
    tol = 2 * bound + 2.0 ** -10 * (h.abs() + want.abs() + b.abs() + o.abs()) + 2.0 ** -24
    if causal:
        m = torch.triu(torch.ones(want.shape[-2:], dtype=torch.bool, device="cuda"), 1)
        want = want.masked_fill(m, -float("inf"))
    return want, tol


def options(store, bias, causal):
    b = TensorView.of(bias)
    s = {"identity": MatmulStore.Identity(), "scale": MatmulStore.Scale(0.125), "add": MatmulStore.Add(),
         "bias": MatmulStore.BetaBias(0.0, b), "beta_bias": MatmulStore.BetaBias(0.5, b),
         "quick_gelu": MatmulStore.QuickGeluBias(b), "beta_gelu": MatmulStore.BetaGeluBias(0.5, b)}[store]
    return MatmulOptions.new().store(s).mask(MatmulMask.Causal if causal else MatmulMask.None_)


# one tile and one k-block; one row, column and k past a tile; the second CTA of a pair without rows or
# columns; fewer k-blocks than stages and more; more tiles than pairs; each store operation
@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (257, 264, 72), (128, 512, 384), (300, 120, 456),
                                   (129, 1000, 1032), (3000, 3080, 200)])
@pytest.mark.parametrize("store,causal,kmajor", [("identity", False, True), ("identity", False, False),
                                                 ("add", False, True), ("bias", False, True), ("beta_bias", False, False),
                                                 ("quick_gelu", False, True), ("scale", True, True), ("beta_gelu", False, False)])
def test_pair_products(kernels, m, n, k, store, causal, kmajor):
    g = torch.Generator(device="cuda").manual_seed(m * 31 + n + k)
    x, w, bias, out0 = half(g, m, k), half(g, k, n), half(g, n), half(g, m, n)
    buf = torch.full((m + 2, n + 16), 5.0, dtype=torch.float16, device="cuda")  # canary around the view
    view = TensorView(buf[1:-1, 8:-8], TensorLayout.new((m, n), (n + 16, 1)))
    buf[1:-1, 8:-8] = out0
    wv = TensorView.of(w.t().contiguous()).permute([1, 0]) if kmajor else TensorView.of(w)
    kernels.set_tunable("tc_pair", 2)
    try:
        kernels.matmul_f16(view, TensorView.of(x), wv, options(store, bias, causal))
    finally:
        kernels.set_tunable("tc_pair", 0)
    assert kernels.last_f16_schedule() == (256, 1, True)
    kernels.device_status()
    want, tol = expected(x, w, out0, bias, store, causal)
    got = buf[1:-1, 8:-8].float()
    live = torch.isfinite(want)
    assert torch.equal(got[~live], want[~live])
    assert bool(((got - want).abs() <= tol)[live].all()), float(((got - want).abs() / tol)[live].max())
    assert bool((buf[0] == 5).all() and (buf[-1] == 5).all() and (buf[:, :8] == 5).all() and (buf[:, -8:] == 5).all())


# batches with both operands strided, one broadcast, and a load-side scale
@pytest.mark.parametrize("bcast", [False, True])
def test_pair_batches(kernels, bcast):
    g = torch.Generator(device="cuda").manual_seed(5)
    B, m, n, k = 3, 290, 328, 136
    x, w = half(g, B, m, k), half(g, 1 if bcast else B, n, k)
    out = torch.zeros((B, m, n), dtype=torch.float16, device="cuda")
    wv = TensorView.of(w[0] if bcast else w).permute([1, 0] if bcast else [0, 2, 1])
    opts = MatmulOptions.new().load(MatmulLoad.Scale(0.5))
    kernels.set_tunable("tc_pair", 2)
    try:
        kernels.matmul_f16(TensorView.of(out), TensorView.of(x), wv, opts)
    finally:
        kernels.set_tunable("tc_pair", 0)
    assert kernels.last_f16_schedule() == (256, 1, True)
    kernels.device_status()
    want, tol = expected(x, w.transpose(1, 2), out, torch.zeros(n, device="cuda"), "identity", False)
    assert bool(((out.float() - 0.25 * want).abs() <= tol).all())


# the store of adr_matmul_nt_f16: one rounding of acc + beta * old
def test_pair_nt_beta(kernels):
    g = torch.Generator(device="cuda").manual_seed(7)
    m, n, k = 300, 520, 200
    x, w, out0 = half(g, m, k), half(g, n, k), half(g, m, n)
    out = out0.clone()
    kernels.set_tunable("tc_pair", 2)
    try:
        kernels.matmul_nt_f16(out, x, w, 0.5)
    finally:
        kernels.set_tunable("tc_pair", 0)
    assert kernels.last_f16_schedule() == (256, 1, True)
    kernels.device_status()
    want = x.float() @ w.float().t() + 0.5 * out0.float()
    tol = (x.float().abs() @ w.float().abs().t()) * (k * 2.0 ** -24) + 2.0 ** -11 * want.abs() + 2.0 ** -24
    assert bool(((out.float() - want).abs() <= tol).all())


# The end of the launch: one fill of the ring of six stages, one fewer than the ring, the whole ring, one more,
# two rounds and one; one tile, or several per pair, which then start anywhere in the ring.  Many launches in a
# row under "pdl", each adding to the output of the one before, so that the next one's CTAs move in as a pair
# leaves: the same bits every time.
@pytest.mark.parametrize("blocks", [1, 5, 6, 7, 13])
@pytest.mark.parametrize("m,n", [(256, 256), (4096, 4608)])
def test_pair_ends(kernels, blocks, m, n):
    g = torch.Generator(device="cuda").manual_seed(blocks)
    x, w, out0 = half(g, m, 64 * blocks), half(g, n, 64 * blocks), half(g, m, n)
    outs, adds = [], 3
    kernels.set_tunable("tc_pair", 2)
    kernels.set_tunable("pdl", 1)
    try:
        for _ in range(10):
            out = out0.clone()
            for _ in range(adds):
                kernels.matmul_f16(TensorView.of(out), TensorView.of(x), TensorView.of(w).permute([1, 0]),
                                   MatmulOptions.new().store(MatmulStore.Add()))
            outs.append(out)
    finally:
        kernels.set_tunable("tc_pair", 0)
        kernels.set_tunable("pdl", 0)
    assert kernels.last_f16_schedule() == (256, 1, True)
    kernels.device_status()
    assert all(torch.equal(o, outs[0]) for o in outs[1:])
    want = out0
    tol = torch.zeros((), device="cuda")
    for _ in range(adds):
        want, step = expected(x, w.t(), want, torch.zeros(n, device="cuda"), "add", False)
        tol = tol + step
    assert bool(((outs[0].float() - want).abs() <= tol).all())


# the same on one CTA per 128 x 256 tile, whose epilogue is compiled for a bias, for bias + QuickGelu, for unaligned
# rows and for the rest: aligned rows that end inside a chunk of 32 columns and beyond a tile, unaligned ones
@pytest.mark.parametrize("m,n,k", [(129, 264, 72), (300, 520, 456), (257, 301, 136)])
@pytest.mark.parametrize("store", ["identity", "add", "bias", "beta_bias", "quick_gelu"])
def test_one_cta_epilogues(kernels, m, n, k, store):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x, w, bias, out0 = half(g, m, k), half(g, n, k), half(g, n), half(g, m, n)
    out = out0.clone()
    tunables = {"tc_bn": 256, "tc_split": 1, "tc_pair": 1}
    for name, value in tunables.items():
        kernels.set_tunable(name, value)
    try:
        kernels.matmul_f16(TensorView.of(out), TensorView.of(x), TensorView.of(w).permute([1, 0]), options(store, bias, False))
    finally:
        for name in tunables:
            kernels.set_tunable(name, 0)
    assert kernels.last_f16_schedule() == (256, 1, False)
    kernels.device_status()
    want, tol = expected(x, w.t(), out0, bias, store, False)
    assert bool(((out.float() - want).abs() <= tol).all())
