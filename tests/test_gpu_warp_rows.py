"""The warp-per-row forms of rms_norm, layer_norm and softmax_rows and the prompt form of RoPE +
cache append, against the library's block-per-row and per-row kernels: the same bits (the orders of
the sums are the same), and against the oracle to one unit in the last place."""
import numpy as np
import pytest
import torch

from adrastea_b200 import TensorLayout, TensorView
from oracle import oracle

pytestmark = pytest.mark.gpu


def bits(t):
    return t.contiguous().view(torch.int16)


def half(rng, *shape, lo=-2.0, hi=2.0):
    return torch.from_numpy(rng.uniform(lo, hi, shape).astype(np.float16)).cuda()


def padded(t, extra):
    """t's rows `extra` elements further apart."""
    buf = torch.full((t.shape[0], t.shape[1] + extra), 7.0, dtype=t.dtype, device=t.device)
    buf[:, :t.shape[1]] = t
    return buf[:, :t.shape[1]]


# one piece; a ragged last chunk; exactly one and just over one register load; several loads; row counts that leave
# the last block partly filled; the last count below the kernels for many rows; the last count at which rms_norm's
# rows of more than 1024 run two to a block, and the first beyond it; rows of any length that cannot be read in
# 16-byte pieces, around the lengths at which their kernels change
@pytest.mark.parametrize("rows,lx", [(1024, 8), (1027, 264), (1026, 1024), (1025, 1032), (1024, 4096), (1025, 4104), (1024, 8192), (1023, 1024),
                                     (1331, 4096), (1332, 4096), (1333, 2048), (1025, 1), (1024, 511), (1027, 513), (1026, 1023),
                                     (1025, 1025), (1500, 2047), (1024, 4095), (1024, 4097)])
def test_norms_same_bits_as_block_kernels(kernels, rows, lx):
    rng = np.random.default_rng(rows * 7919 + lx)
    x, w, b = half(rng, rows, lx), half(rng, lx, lo=0.5, hi=1.5), half(rng, lx, lo=-0.5, hi=0.5)
    T = TensorView.of

    def both(x, o1, o2):
        kernels.rms_norm(T(o1), T(x), T(w), 1e-5)
        kernels.layer_norm(T(o2), T(x), T(w), T(b), 1e-5)

    want = [torch.zeros_like(x) for _ in range(2)]
    for part in (slice(0, rows // 2), slice(rows // 2, rows)):  # fewer than 1024 rows: a block per row
        both(x[part], *(t[part] for t in want))
    for xp, pad in ((x, 0), (padded(x, 8), 16), (padded(x, 1), 1)):  # 16-byte rows, wider pitches, an odd pitch
        got = [padded(torch.zeros_like(x), pad) for _ in range(2)]
        both(xp, *got)
        assert all(torch.equal(bits(g), bits(t)) for g, t in zip(got, want))


# one element; around the 32-lane and the 256-thread boundaries; the last width of each form and
# the first that stays with the block-per-row kernel; few rows and enough for the warp-per-row kernel
@pytest.mark.parametrize("w", [1, 31, 33, 256, 257, 512, 513, 1024, 1025])
@pytest.mark.parametrize("temp", [1.0, 0.7])
@pytest.mark.parametrize("rows", ["few", "many"])
def test_softmax_rows(kernels, w, temp, rows):
    rng = np.random.default_rng(w)
    x = (rng.standard_normal((3, 11 if rows == "few" else (2 * w + 2) // 3, w)) * 3).astype(np.float16)
    x[0, 0, w // 2:] = -np.inf if w > 1 else 0
    o = torch.from_numpy(x.copy()).cuda()
    kernels.softmax_rows_inplace(TensorView.of(o), temp)
    want = oracle.softmax_rows(x, temp=temp)
    got = o.cpu().numpy()
    d = np.abs(got.view(np.uint16).astype(np.int32) - want.view(np.uint16).astype(np.int32))
    assert d.max() <= 1 and (d != 0).mean() < 0.02 + 2.0 / d.size


def test_softmax_of_more_rows_than_a_grid_holds(kernels):
    """65535 heads of 262152 rows of one element, 34 GB: over 2^34 rows, where a grid of four rows per block
    holds 2^33.  A row of one element becomes 1 (the buffer is looked at four elements at a time)."""
    heads, h = 65535, 262152
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB")
    x = torch.zeros(heads * h, dtype=torch.float16, device="cuda")
    kernels.softmax_rows_inplace(TensorView(x, TensorLayout.new((heads, h, 1), (h, 1, 1))))
    lo, hi = torch.aminmax(x.view(torch.int64))
    assert int(lo) == int(hi) == 0x3C003C003C003C00


def test_softmax_same_bits_as_block_kernel(kernels):
    """A row of 1100 with -inf behind element w is summed over the same elements in the same order by
    the block-per-row kernel (exp(-inf) adds +0)."""
    rng = np.random.default_rng(3)
    for w, rows in ((40, 64), (257, 513), (257, 514), (512, 1024), (700, 1199), (700, 1200), (1024, 1200)):
        x = torch.full((rows, 1100), -float("inf"), dtype=torch.float16, device="cuda")
        x[:, :w] = half(rng, rows, w, lo=-6, hi=6)
        y = x.clone()
        kernels.softmax_rows_inplace(TensorView.of(x))
        kernels.softmax_rows_inplace(TensorView(y, TensorLayout.new((rows, w), (1100, 1))))
        assert torch.equal(bits(x[:, :w]), bits(y[:, :w]))
        assert bool((y[:, w:] == -float("inf")).all())


# one head and many; head sizes of a single piece and the largest; batches around the number of
# sequences of a block; a prompt shorter than the cache
@pytest.mark.parametrize("B,T,heads,hd,S", [(1, 3, 1, 8, 3), (4, 5, 4, 64, 9), (5, 2, 3, 128, 8), (9, 1, 2, 256, 1), (2, 7, 33, 80, 16)])
def test_prefill_rope_append(kernels, B, T, heads, hd, S):
    rng = np.random.default_rng(B * T + hd)
    width = heads * hd
    qkv = half(rng, B * T, 3 * width + 8)
    ref = qkv.clone()
    kc = torch.full((B, S, width), 3.0, dtype=torch.float16, device="cuda")
    vc = kc.clone()
    q, k, v = (qkv[:, i * width:(i + 1) * width] for i in range(3))
    T_ = TensorView.of
    kernels.prefill_rope_append(T_(q), T_(k), T_(v), kc, vc, T, heads, 10000.0)
    rq, rk = ref[:, :width], ref[:, width:2 * width]
    for b in range(B):
        for t in (rq, rk):
            kernels.rotary_inplace(T_(t[b * T:(b + 1) * T]), heads, 0, 10000.0)
    assert torch.equal(bits(q), bits(rq))
    assert torch.equal(bits(kc[:, :T]), bits(rk.reshape(B, T, width)))
    assert torch.equal(bits(vc[:, :T]), bits(v.reshape(B, T, width)))
    assert torch.equal(bits(v), bits(ref[:, 2 * width:3 * width]))
    assert bool((kc[:, T:] == 3.0).all()) and bool((vc[:, T:] == 3.0).all())
