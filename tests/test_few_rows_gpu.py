"""The few-rows product at every count of eights of tokens it has a kernel for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 8, 9, 17, 24, 25, 32, 33, 40, 41, 48, 49, 56, 57, 64])
@pytest.mark.parametrize("N,K", [(70, 72), (512, 2560)])
def test_rows_by_eights(M, N, K):
    """Against 64-bit, and a row the same whatever the rows beside it within one cut of K: the kernels differ in their rows alone."""
    from gopherllm_b200 import ops as o
    g = torch.Generator().manual_seed(M)
    a = torch.randn(64, K, generator=g).bfloat16()
    w = (torch.randn(N, K, generator=g) * K ** -0.5).bfloat16()
    bias, add = torch.randn(N, generator=g), torch.randn(64, N, generator=g)
    want = a.double() @ w.double().T + bias.double() + add.double()
    ad, wd, bd, xd = a.cuda(), w.cuda(), bias.cuda(), add.cuda()
    for split in (1, 4):
        got = o.gemm_skinny(ad[:M], wd, bd, None, xd[:M], out_dtype=torch.float32, split_k=split)
        # K exact products summed in 32 bits: K / 2 roundings of 2^-24 of the partial sums at most
        assert (got.double().cpu() - want[:M]).abs().max() <= K * 2 ** -24 * max(1.0, float(want.abs().max()))
        whole = o.gemm_skinny(ad, wd, bd, None, xd, out_dtype=torch.float32, split_k=split)
        assert torch.equal(got, whole[:M])
    assert o.wait_failures()["libgl_gemm_skinny"] == 0, "a bounded wait ran out"
