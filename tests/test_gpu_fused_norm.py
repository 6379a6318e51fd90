"""rms_norm inside the decode products: the bits of the norm's own kernel followed by the product."""
import pytest
import torch

from adrastea_b200 import Kernel, TensorView

pytestmark = pytest.mark.gpu


# fewer elements than threads; rows that end inside a pass of the threads; more weights than are requested
# ahead; one to sixteen rows, on both sides of the lines between all threads and a warp for a row (three rows, 1024
# elements for each); ragged n; both kinds of zero point
@pytest.mark.parametrize("m,p,n,bs,zp", [(1, 128, 48, 64, False), (1, 4096, 11008, 128, False), (4, 1280, 333, 64, True),
                                         (3, 8448, 100, 64, False), (2, 11008, 64, 128, False), (8, 2048, 250, 128, False),
                                         (5, 768, 16, 128, True), (9, 1280, 48, 64, False), (16, 4096, 100, 128, True),
                                         (4, 4096, 64, 128, False), (4, 4224, 48, 64, False), (7, 8192, 32, 128, False),
                                         (8, 8192, 32, 64, False)])
def test_norm_inside_the_decode_products(kernels, m, p, n, bs, zp):
    g = torch.Generator(device="cuda").manual_seed(m * p + n)
    x = (torch.randn((m, p), device="cuda", generator=g) * torch.rand((m, 1), device="cuda", generator=g) * 3).half()
    w = (torch.rand(p, device="cuda", generator=g) + 0.5).half()
    q = torch.randint(0, 256, (2 * n, p), dtype=torch.uint8, device="cuda", generator=g)
    s = (torch.rand((2 * n, p // bs), device="cuda", generator=g) * 0.009 + 0.001).half()
    z = (torch.rand((2 * n, p // bs), device="cuda", generator=g) * 16 + 120).half() if zp else None
    zg, zu = (z[:n], z[n:]) if zp else (None, None)
    old = torch.randn((m, n), device="cuda", generator=g).half()
    xn = torch.zeros_like(x)
    kernels.rms_norm(TensorView.of(xn), TensorView.of(x), TensorView.of(w), 1e-5)
    two, two_silu = old.clone(), torch.zeros_like(old)
    kernels.force_kernel(Kernel.U8Ring)
    try:
        kernels.matmul_nt_fp16u8(two, xn, q[:n], s[:n], bs, 0.5, zg)
    finally:
        kernels.force_kernel(Kernel.Auto)
    paired = m <= 8  # more rows: the paired product has no norm
    if paired:
        kernels.silu_mul_matmul_nt_fp16u8(two_silu, xn, q[:n], s[:n], q[n:], s[n:], bs, zg, zu)
    for pdl in (0, 1):
        kernels.set_tunable("pdl", pdl)
        try:
            one, one_silu = old.clone(), torch.full_like(old, 7.0)
            kernels.rms_norm_matmul_nt_fp16u8(one, x, w, 1e-5, q[:n], s[:n], bs, 0.5, zg)
            if paired:
                kernels.silu_mul_matmul_nt_fp16u8(one_silu, x, q[:n], s[:n], q[n:], s[n:], bs, zg, zu, norm_weights=w,
                                                  eps=1e-5)
        finally:
            kernels.set_tunable("pdl", 0)
        torch.cuda.synchronize()
        kernels.device_status()
        assert torch.equal(one, two) and (not paired or torch.equal(one_silu, two_silu))
