"""32-bit attention with several rows a warp: the same numbers as a row a warp, and as 64-bit says."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,hd", [(2, 2, 4), (4, 2, 64), (3, 1, 36), (2, 2, 100), (2, 1, 256), (2, 2, 50)])
@pytest.mark.parametrize("window", [0, 40])
def test_rows_do_not_depend_on_the_rows_beside_them(H, G, hd, window, dtype):
    """Runs that end inside a warp's rows, a block's and a page, behind nothing and behind cached positions: in one call, in calls
    of at most eight rows and of one, bit for bit; and against 64-bit."""
    from gopherllm_b200 import ops
    g = torch.Generator().manual_seed(hd + window)
    qlens, ctxs = [37, 1, 9, 70], [0, 130, 61, 300]
    B, T = len(qlens), sum(qlens)
    totals = [c + q for c, q in zip(ctxs, qlens)]
    most = max(-(-n // 64) for n in totals)
    pages, at = torch.zeros(B, most, dtype=torch.int32), 0
    for b, n in enumerate(totals):
        k = -(-n // 64)
        pages[b, :k] = torch.arange(at, at + k).flip(0)
        at += k
    keys, values = (torch.full((at, G, 64, hd), float("nan"), dtype=dtype) for _ in range(2))
    for b, n in enumerate(totals):
        for j in range(n):
            for t in (keys, values):
                t[pages[b, j // 64], :, j % 64] = torch.randn(G, hd, generator=g).to(dtype)
    q = (torch.randn(T, H * hd, generator=g) * hd ** -0.5).to(dtype)
    kd, vd, pd = keys.cuda(), values.cuda(), pages.cuda()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731

    def call(runs):
        """runs: (sequence, first row of its run, rows); their results in order"""
        rows = torch.cat([q[sum(qlens[:b]) + r:sum(qlens[:b]) + r + n] for b, r, n in runs]).cuda()
        out = torch.empty_like(rows)
        lens = [n for _, _, n in runs]
        ops.attention_generic(rows, out, kd, vd, i32([sum(lens[:i]) for i in range(len(runs))]), i32(lens),
                              i32([ctxs[b] + r for b, r, _ in runs]), pd[[b for b, _, _ in runs]].contiguous(), H, G, hd, max(lens), window)
        return out.cpu()

    whole = call([(b, 0, n) for b, n in enumerate(qlens)])
    for b, n in enumerate(qlens):
        mine = whole[sum(qlens[:b]):sum(qlens[:b]) + n]
        assert torch.equal(call([(b, 0, n)]), mine)
        if n > 1:                                            # (rows of a longer run and a lone token have forms of their own)
            assert torch.equal(torch.cat([call([(b, r, min(8, n - r))]) for r in range(0, n - 1, 8)])[:n - 1], mine[:n - 1])
        for r in range(n):
            p = ctxs[b] + r
            lo = max(0, p - window + 1) if window else 0
            k, v = (torch.stack([t[pages[b, j // 64], :, j % 64] for j in range(lo, p + 1)]).double() for t in (keys, values))
            k, v = (t.repeat_interleave(H // G, 1) for t in (k, v))
            s = torch.softmax(torch.einsum("hd,jhd->hj", q[sum(qlens[:b]) + r].double().view(H, hd), k), -1)
            want = torch.einsum("hj,jhd->hd", s, v).reshape(-1)
            # scores and weighted values: up to 370 products of 2^-24 each, and the result's rounding
            eps = 370 * 2 ** -24 * 4 + (2 ** -8 if dtype == torch.bfloat16 else 0.0)
            assert ((mine[r].double() - want).abs() <= eps * max(1.0, float(want.abs().max()))).all(), (b, r)
