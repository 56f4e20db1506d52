"""The 32-bit attention kernels: one, two and four rows a warp and a lone token's forms give the same numbers, and what 64-bit says."""
import ctypes

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


def paged_call(H, G, hd, dtype, qlens, ctxs, window, seed):
    """Sequences on pages in any order, NaN where nothing was written; the call over parts of them, and all results in 64-bit."""
    from gopherllm_b200 import ops
    g = torch.Generator().manual_seed(seed)
    totals = [c + q for c, q in zip(ctxs, qlens)]
    most, at = max(-(-n // 64) for n in totals), 0
    pages = torch.zeros(len(qlens), most, dtype=torch.int32)
    for b, n in enumerate(totals):
        k = -(-n // 64)
        pages[b, :k] = torch.arange(at, at + k).flip(0)
        at += k
    kv = torch.randn(2, sum(totals), G, hd, generator=g).to(dtype)
    cache = torch.full((2, at, G, 64, hd), float("nan"), dtype=dtype)
    q = (torch.randn(sum(qlens), H * hd, generator=g) * hd ** -0.5 * 3).to(dtype)
    want = torch.empty(sum(qlens), H * hd, dtype=torch.float64)
    for b, n in enumerate(totals):
        mine = kv[:, sum(totals[:b]):sum(totals[:b]) + n]
        j = torch.arange(n)
        cache[:, pages[b, j // 64].long(), :, j % 64] = mine.transpose(0, 1)
        k, v = (t.double().repeat_interleave(H // G, 1) for t in mine)
        p, rows = torch.arange(ctxs[b], n), slice(sum(qlens[:b]), sum(qlens[:b + 1]))
        s = torch.einsum("thd,jhd->htj", q[rows].double().view(-1, H, hd), k)
        hidden = (j[None] > p[:, None]) | ((j[None] <= p[:, None] - window) if window else torch.zeros(1, 1, dtype=torch.bool))
        want[rows] = torch.einsum("htj,jhd->thd", torch.softmax(s.masked_fill(hidden, float("-inf")), -1), v).reshape(-1, H * hd)
    kd, vd, pd = cache[0].cuda(), cache[1].cuda(), pages.cuda()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731

    def call(runs):
        """runs: (sequence, first row of its run, rows); the results in order, and the form the call took"""
        rows = torch.cat([q[sum(qlens[:b]) + r:sum(qlens[:b]) + r + n] for b, r, n in runs]).cuda()
        out, lens = torch.empty_like(rows), [n for _, _, n in runs]
        args = (rows, out, kd, vd, i32([sum(lens[:i]) for i in range(len(runs))]), i32(lens), i32([ctxs[b] + r for b, r, _ in runs]),
                pd[[b for b, _, _ in runs]].contiguous(), H, G, hd)
        ops.attention_generic(*args, max(lens), window)
        form = ops._lib("attention_generic.cu").gl_attention_generic_rows(ctypes.byref(ops._attn_args(*args, window, max(lens), 1.0)),
                                                                          ctypes.c_int(ops.dtype_code(dtype)))
        return out.cpu(), form
    return call, want


def close(got, want, dtype, keys):
    # scores and weighted values: as many products of 2^-24 each, and the result's rounding
    eps = keys * 2 ** -24 * 4 + (2 ** -8 if dtype == torch.bfloat16 else 0.0)
    assert ((got.double() - want).abs() <= eps * max(1.0, float(want.abs().max()))).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,hd", [(16, 4, 64), (16, 2, 36), (16, 16, 128), (16, 4, 256)])
@pytest.mark.parametrize("window", [0, 40])
def test_one_two_and_four_rows_a_warp(H, G, hd, window, dtype):
    """The same rows in calls that take four rows a warp, two and one, bit for bit."""
    qlens, ctxs = [37, 1, 9, 300], [0, 130, 61, 20]
    call, want = paged_call(H, G, hd, dtype, qlens, ctxs, window, hd)
    whole, form = call([(b, 0, n) for b, n in enumerate(qlens)])
    assert form == 4
    close(whole, want, dtype, 330)
    long = whole[sum(qlens[:3]):]
    half, form = call([(3, 0, 150)])
    assert form == 2 and torch.equal(half, long[:150])
    for r in range(0, 300, 8):
        few, form = call([(3, r, min(8, 300 - r))])
        assert form == 1 and torch.equal(few, long[r:r + 8])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,hd", [(8, 2, 64), (8, 8, 36), (8, 2, 96), (8, 1, 128), (4, 4, 256)])
@pytest.mark.parametrize("window", [0, 300])
def test_lone_tokens_alone_in_a_crowd_and_beside_a_prompt(H, G, hd, window, dtype):
    """One token of each of many sequences, whose pages make whole rounds of a block's warps, half ones and neither: the same
    numbers as alone and as beside a prompt, and those of 64-bit."""
    ctxs = [0, 63, 190, 191, 192, 255, 256, 319, 320, 511, 512, 639, 700, 900] * 3
    n = len(ctxs)
    call, want = paged_call(H, G, hd, dtype, [1] * n + [20], ctxs + [5], window, hd + 1)
    crowd, form = call([(b, 0, 1) for b in range(n)])
    assert form == (0 if dtype == torch.bfloat16 and hd <= 96 else 1)
    close(crowd, want[:n], dtype, 900)
    beside, form = call([(b, 0, 1) for b in range(n)] + [(n, 0, 20)])
    assert form > 0 and torch.equal(beside[:n], crowd)
    for b in range(14):
        alone, form = call([(b, 0, 1)])
        assert form == 1 and torch.equal(alone, crowd[b:b + 1]), ctxs[b]
