"""The norm of many rows, a warp or a block a row: its sums in the order of a warp that holds the row, its result to the last bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
F, D64 = np.float32, np.float64


def fma(a, b, c):
    """a * b + c rounded once (the product of two 32-bit numbers is exact in 64)"""
    return (a.astype(D64) * b.astype(D64) + c.astype(D64)).astype(F)


def row_sums(pieces):
    """[R, n] -> [R]: lane l of 32 adds pieces l, l + 32, ... in turn, then the lanes are added crosswise, 16, 8, 4, 2 and 1 apart."""
    R, n = pieces.shape
    lanes = np.zeros((R, 32), F)
    for k in range(0, n, 32):
        part = pieces[:, k:k + 32]
        lanes[:, :part.shape[1]] = lanes[:, :part.shape[1]] + part
    for o in (16, 8, 4, 2, 1):
        lanes = lanes + lanes[:, np.arange(32) ^ o]
    return lanes[:, 0]


def statistics(x, eps, rms):
    """mean and factor of every row, as 32-bit numbers"""
    R, D = x.shape
    p = x.reshape(R, D // 4, 4)
    mean = np.zeros(R, F) if rms else row_sums((p[..., 0] + p[..., 1]) + (p[..., 2] + p[..., 3])) / F(D)
    c = p - mean[:, None, None]
    var = row_sums(fma(c[..., 0], c[..., 0], c[..., 1] * c[..., 1]) + fma(c[..., 2], c[..., 2], c[..., 3] * c[..., 3])) / F(D)
    return mean, (1.0 / np.sqrt((var + F(eps)).astype(D64))).astype(F)


# one, two and four pieces a thread, a piece short of and over each, one piece a row, the longest row it takes
# rows taken by blocks, and (4,100) by warps
@pytest.mark.parametrize("R", [257, 4100])
@pytest.mark.parametrize("D", [4, 128, 252, 256, 260, 508, 512, 516, 2044, 2560, 4092, 4096])
@pytest.mark.parametrize("rms,bias,gather", [(False, True, False), (True, False, False), (False, False, True), (True, True, True)])
def test_norm_of_many_rows(D, rms, bias, gather, R):
    from gopherllm_b200 import ops
    g = torch.Generator().manual_seed(D)
    N = R + (43 if gather else 0)
    x = torch.randn(N, D, generator=g) * (0.1 + 3.0 * torch.rand(N, 1, generator=g)) + 0.5
    gamma, beta = 1.0 + 0.1 * torch.randn(D, generator=g), torch.randn(D, generator=g) if bias else None
    rows = torch.randperm(N, generator=g)[:R] if gather else None
    got = ops.norm(x.cuda(), gamma.cuda(), None if beta is None else beta.cuda(), 1e-5, torch.bfloat16,
                   rms, None if rows is None else rows.int().cuda()).cpu()
    some = slice(None, None, 1 if R < 300 else 13)
    x, got = (x[rows] if gather else x)[some], got[some]
    want = x.double() - (0.0 if rms else x.double().mean(-1, keepdim=True))
    want = want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-5) * gamma.double() + (beta.double() if bias else 0.0)
    # one rounding to 8 bits (half a unit: 2^-8), behind a few to 24 of numbers of the row's size
    assert ((got.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5 * want.abs().max()).all()
    mean, inv = statistics(x.numpy(), 1e-5, rms)
    unit = (x.numpy() - mean[:, None]) * inv[:, None]
    y = unit * gamma.numpy() + (beta.numpy() if bias else F(0))
    assert torch.equal(got, torch.from_numpy(y).bfloat16())
