"""The vectorised quantiser against the oracle and against the library's warp-per-group kernel
(which any buffer that is not 16-byte aligned reaches): whole codes and scale bits, no tolerance."""
import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


def shifted(t):
    """A copy of t that starts 2 bytes past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    v = buf[1:1 + t.numel()].view(t.shape)
    v.copy_(t)
    return v


# small tensors and blocks of 48 and 1024, which the warp-per-group kernel takes; the last of these; beyond them
# lanes per group 1, 2, 4, 8, 16, 32, with groups that leave a warp and a block partly filled
@pytest.mark.parametrize("rows,k,bs", [(1, 16, 16), (3, 96, 32), (5, 192, 64), (7, 640, 128), (129, 768, 256),
                                       (9, 1024, 512), (4, 96, 48), (2, 2048, 1024), (4096, 16, 16), (2048, 512, 512),
                                       (4097, 16, 16), (2049, 64, 32), (1367, 192, 64), (821, 640, 128),
                                       (1367, 768, 256), (2049, 512, 512)])
def test_quantize_codes(kernels, rows, k, bs):
    rng = np.random.default_rng(rows * k + bs)
    x = (rng.standard_normal((rows, k)) * rng.uniform(0.01, 2.0, (rows, 1))).astype(np.float16)
    x[0, :bs] = 0                                    # scale 0
    x[-1, ::3] = 0                                   # ties: 127.5 rounds away from zero
    x[-1, 1] = 4.0
    # sums on and next to half-integers: multiples of the group's own scale
    x[rows // 2, -bs:] = (np.arange(bs) % 255 - 127).astype(np.float16) * np.float16(0.03125)
    x[rows // 2, -1] = np.float16(127.5 * 0.03125)
    bits = rng.integers(0, 1 << 16, (rows, k), dtype=np.uint16).view(np.float16)  # NaN, inf, subnormals
    tiny = rng.integers(0, 1 << 8, (rows, k), dtype=np.uint16).view(np.float16)   # subnormal scales
    for data in (x, bits, tiny):
        xd = torch.from_numpy(data.copy()).cuda()
        q = torch.full((rows, k), 77, dtype=torch.uint8, device="cuda")
        s = torch.zeros((rows, k // bs), dtype=torch.float16, device="cuda")
        q2, s2 = torch.full_like(q, 78), torch.zeros_like(s)
        kernels.quantize_absmax_uint8(q, s, xd)
        kernels.quantize_absmax_uint8(q2, s2, shifted(xd))
        torch.cuda.synchronize()
        assert torch.equal(s.view(torch.int16), s2.view(torch.int16))
        assert torch.equal(q, q2)
        if data is x:
            wq, ws = oracle.quantize(x, bs)
            assert np.array_equal(s.cpu().numpy().view(np.uint16), ws.view(np.uint16))
            live = np.repeat(ws != 0, bs, axis=1)  # 0 / 0 has no defined code
            assert np.array_equal(q.cpu().numpy()[live], wq[live])
