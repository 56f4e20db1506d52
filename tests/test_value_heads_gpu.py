"""Attention with a table over the heads: blocks of one, two and four value heads give the same numbers."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


# (key size, value size, query heads, value heads, value heads a block in the joint call)
@pytest.mark.parametrize("hd,vd,H,G,most", [(64, 64, 16, 4, 4), (32, 32, 24, 6, 2), (64, 32, 16, 8, 4), (96, 96, 16, 4, 2), (128, 64, 24, 6, 2),
                                            (256, 64, 8, 4, 2), (256, 192, 8, 4, 1)])
def test_value_heads_a_block(hd, vd, H, G, most):
    """Runs that end inside a tile, behind nothing and behind cached positions: all in one call, which has blocks enough for several
    value heads each, and one by one, which has not; bit for bit, and against 64-bit."""
    import ctypes
    from gopherllm_b200 import ops
    from gopherllm_b200.csrc import catalog
    g = torch.Generator().manual_seed(hd + vd)
    qlens, ctxs = [100, 2, 64, 65, 130] * 5, [0, 70, 3, 0, 40] * 5
    totals = [c + q for c, q in zip(ctxs, qlens)]
    B, per = len(qlens), 3
    pages = torch.randperm(B * per, generator=g).int().view(B, per)
    k, v = torch.randn(sum(totals), G, hd, generator=g).bfloat16(), torch.randn(sum(totals), G, vd, generator=g).bfloat16()
    kc, vc = torch.zeros(B * per, G, 64, hd, dtype=torch.bfloat16), torch.zeros(B * per, G, 64, vd, dtype=torch.bfloat16)
    q = torch.randn(sum(qlens), H * hd, generator=g).bfloat16()
    mix = torch.eye(H) + 0.2 * torch.randn(H, H, generator=g)
    for b, n in enumerate(totals):
        j, at = torch.arange(n), sum(totals[:b])
        kc[pages[b, j // 64].long(), :, j % 64], vc[pages[b, j // 64].long(), :, j % 64] = k[at:at + n], v[at:at + n]
    kc, vc, pages, mixed = kc.cuda(), vc.cuda(), pages.cuda(), mix.cuda()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    lib = ops._lib("attention_mixed_tc.cu", catalog.pair_dim_defines(hd, vd))

    def call(seqs):
        lens = [qlens[b] for b in seqs]
        ctx = SimpleNamespace(seq_qstart=i32([sum(lens[:i]) for i in range(len(lens))]), seq_qlen=i32(lens), seq_ctx=i32([ctxs[b] for b in seqs]),
                              n_seqs=len(lens), max_qlen=max(lens), max_len=max(totals), n_tokens=sum(lens))
        rows = torch.cat([q[sum(qlens[:b]):sum(qlens[:b + 1])] for b in seqs]).cuda()
        a = ops._PairsArgs()
        a.B, a.nH, a.nVal, a.max_qlen, a.T = len(lens), H, G, max(lens), sum(lens)
        return ops.attention_mixed(rows, kc, vc, ctx, pages[seqs].contiguous(), H, G, hd, vd, mix=mixed, score_scale=hd ** -0.5).cpu(), \
            lib.gl_attention_pairs_tc_heads(ctypes.byref(a))

    whole, heads = call(list(range(B)))
    assert heads == most
    for b in range(5):
        rows = slice(sum(qlens[:b]), sum(qlens[:b + 1]))
        alone, heads = call([b])
        assert heads == 1
        assert torch.equal(alone, whole[rows]), b
        at, n, p = sum(totals[:b]), totals[b], torch.arange(ctxs[b], totals[b])
        s = torch.einsum("thd,jhd->htj", q[rows].double().view(-1, H, hd), k[at:at + n].double().repeat_interleave(H // G, 1)) * hd ** -0.5
        w = torch.softmax(s.masked_fill(torch.arange(n)[None] > p[:, None], float("-inf")), -1)
        w = torch.einsum("hg,gtj->htj", mix.double(), w)
        want = torch.einsum("htj,jhd->thd", w, v[at:at + n].double().repeat_interleave(H // G, 1)).reshape(len(p), -1)
        # weights rounded to bfloat16 before they meet the values, the result once more; as many as the table's row adds up
        bound = 2 ** -8 * float(mix.abs().sum(-1).max()) * float(v.abs().max())
        assert (whole[rows].double() - want).abs().max() <= bound
