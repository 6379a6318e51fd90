"""Chains of kernels that start before the launch ahead of them has ended ("pdl"), each on the result of the
one before and over buffers that the one before still reads: the bits of the same chain run one by one."""
import pytest
import torch

from adrastea_b200 import MatmulOptions, MatmulStore, TensorLayout, TensorView

pytestmark = pytest.mark.gpu


# one tile; a k-split; a last wave on clusters behind full waves (150 tiles of 128 x 256); CTA pairs
@pytest.mark.parametrize("tokens,width,wide", [(40, 256, 384), (257, 512, 1536), (768, 1024, 6400), (2048, 512, 4096)])
def test_chains(kernels, tokens, width, wide):
    g = torch.Generator(device="cuda").manual_seed(tokens)
    half = lambda *s: (torch.randn(s, device="cuda", generator=g) * 0.05).half()
    x0, w1, bias = half(tokens, width) * 20, half(wide, width), half(wide)
    q = torch.randint(0, 256, (wide, width), dtype=torch.uint8, device="cuda", generator=g)
    s = (torch.rand((wide, width // 128), device="cuda", generator=g) * 1e-3 + 1e-4).half()
    wd = half(width, wide)
    heads = TensorLayout.new((4, tokens, 64), (64, width, 1))

    schedules = set()

    def product(*args):
        kernels.matmul_f16(*args)
        schedules.add(kernels.last_f16_schedule())

    def chain():
        x, f = x0.clone(), torch.zeros((wide, width), dtype=torch.float16, device="cuda")
        h, u = (torch.zeros((tokens, wide), dtype=torch.float16, device="cuda") for _ in range(2))
        p = torch.zeros((4, tokens, tokens), dtype=torch.float16, device="cuda")
        for _ in range(6):
            kernels.matmul_nt_fp16u8(u, x, q, s, 128, 0.5)
            kernels.dequantize_absmax_uint8(f, s, q)
            product(TensorView.of(h), TensorView.of(x), TensorView.of(f).permute([1, 0]),
                    MatmulOptions.new().store(MatmulStore.BetaBias(0.5, TensorView.of(bias))))
            product(TensorView.of(h), TensorView.of(x), TensorView.of(w1).permute([1, 0]),
                    MatmulOptions.new().store(MatmulStore.Add()))
            product(TensorView.of(u), TensorView.of(x), TensorView.of(w1).permute([1, 0]),
                    MatmulOptions.new().store(MatmulStore.Add()))
            product(TensorView.of(x), TensorView.of(h), TensorView.of(wd).permute([1, 0]))
            v = TensorView(x, heads)
            product(TensorView.of(p), v, v.permute([0, 2, 1]), MatmulOptions.new().store(MatmulStore.Scale(0.125)))
            kernels.softmax_rows_inplace(TensorView.of(p))
            o = TensorView(h, TensorLayout.new((4, tokens, 64), (64, wide, 1)))
            product(o, TensorView.of(p), v)
            kernels.attention_f16(v, o, o, o, 0.125)
        return x, h, u, p

    want = chain()
    torch.cuda.synchronize()
    if tokens == 257:
        assert any(split > 1 for _, split, _ in schedules)
    if tokens == 2048:
        assert any(pair for _, _, pair in schedules)
    kernels.set_tunable("pdl", 1)
    try:
        for _ in range(3):
            got = chain()
            torch.cuda.synchronize()
            kernels.device_status()
            assert all(torch.equal(a.view(torch.int16), b.view(torch.int16)) for a, b in zip(got, want))
    finally:
        kernels.set_tunable("pdl", 0)
