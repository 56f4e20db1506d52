"""The kernels over 32-bit rows, by 16-byte pieces and element by element, against 64-bit, at the edges of their shapes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def close(got, want, eps):
    """eps: what the result's type and the sum over a row round, relative to a result of the row's size."""
    err = (got.double().cpu() - want).abs()
    assert bool((err <= eps * want.abs().clamp(min=1.0)).all()), float(err.max())


# pieces a thread of 1, 2, 4 and 8, a piece short and over; rows that are no whole pieces, and rows longer than the kernels by pieces take
@pytest.mark.parametrize("D", [4, 30, 64, 256, 260, 1024, 1028, 2048, 2052, 4096, 4100, 8192, 8196])
@pytest.mark.parametrize("R", [1, 63, 64])
def test_row_norms(R, D):
    from gopherllm_b200 import ops as o
    g = torch.Generator().manual_seed(D + R)
    a, b, c, d, e = (torch.randn(R, D, generator=g, dtype=torch.float64).float() for _ in range(5))
    w1, w2 = (1.0 + 0.1 * torch.randn(D, generator=g, dtype=torch.float64) for _ in range(2))
    w1, w2 = w1.float(), w2.float()
    dev = [t.cuda() for t in (a, b, c, d, e)]
    W1, W2 = w1.cuda(), w2.cuda()
    unit = lambda x: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6)  # noqa: E731
    A, B, C, D2, E2, v1, v2 = (t.double() for t in (a, b, c, d, e, w1, w2))
    f32, b16 = 2e-6 * 4, 2 ** -8                     # sums of up to 8,196 squares in parts: a few units in the last place
    for dtype, eps in ((torch.float32, f32), (torch.bfloat16, b16)):
        x1, x2 = o.rms_norm_pair(dev[0], W1, W2, 1e-6, dtype)
        close(x1, unit(A) * v1, eps)
        close(x2, unit(A) * v2, eps)
    for adds in ([], [2], [2, 3], [2, 3, 4]):
        extra = sum(((C, D2, E2)[i - 2] for i in adds), torch.zeros_like(A))
        close(o.rms_scale_add(dev[0], W1, 1e-6, 0.5, adds=[dev[i] for i in adds]), 0.5 * unit(A) * v1 + extra, f32 * 2)
        close(o.rms_scale_add(dev[0], W1, 1e-6, 0.5, adds=[dev[i] for i in adds], second=(dev[1], W2)),
              0.5 * unit(A) * v1 + 0.5 * unit(B) * v2 + extra, f32 * 2)
    out = dev[2].clone()                             # onto one of the adds
    o.rms_scale_add(dev[0], W1, 1e-6, 1.0, adds=[dev[3], out], out=out)
    close(out, unit(A) * v1 + C + D2, f32 * 2)
    out, copy = o.post_norm_add(dev[0], W1, 1e-6, dev[2], scale=0.7)
    assert copy is None
    close(out, C + unit(0.7 * A) * v1, f32)
    out = dev[2].clone()
    _, copy = o.post_norm_add(dev[0], W1, 1e-6, out, out=out, scale=0.7, second=(dev[1], -1.3), rounded=torch.bfloat16)
    want = C + unit(0.7 * A - 1.3 * B) * v1
    close(out, want, f32)
    close(copy, want, b16)
    assert torch.equal(copy, out.bfloat16())


# 8, 16 and 32 lanes an item and up to 8 pieces a lane; items that leave a block part empty; gates that are no whole pieces
@pytest.mark.parametrize("H,V", [(1, 4), (3, 32), (5, 36), (8, 64), (7, 100), (8, 128), (3, 256), (8, 512), (2, 640), (1, 1024), (1, 1028), (4, 30)])
@pytest.mark.parametrize("off", [0, 8, 2])
def test_head_norm_gate(H, V, off):
    from gopherllm_b200 import ops as o
    g = torch.Generator().manual_seed(H * V + off)
    for T in (1, 5):
        x = torch.randn(T, H * V, generator=g)
        xd = x.cuda()
        unit = lambda t: t / torch.sqrt((t * t).mean(-1, keepdim=True) + 1e-6)  # noqa: E731
        for dtype, eps in ((torch.float32, 8e-6), (torch.bfloat16, 2 ** -7)):
            gate = torch.randn(T, off + H * V + 6, generator=g).to(dtype)
            z = gate.double()[:, off:off + H * V].reshape(T, H, V)
            for w in (None, torch.randn(V, generator=g), torch.randn(H * V, generator=g)):
                W = torch.ones(H, V).double() if w is None else w.double().reshape(-1, V).expand(H, V)
                wd = None if w is None else w.cuda()
                X = x.double().reshape(T, H, V)
                close(o.head_norm_gate(xd, wd, H, V, 1e-6, dtype).reshape(T, H, V), unit(X) * W, eps)
                for act, s in (("sigmoid", torch.sigmoid(z)), ("silu", z * torch.sigmoid(z))):
                    kw = dict(gate=gate.cuda(), gate_off=off, gate_act=act)
                    close(o.head_norm_gate(xd, wd, H, V, 1e-6, dtype, **kw).reshape(T, H, V), unit(X) * W * s, eps)
                    close(o.head_norm_gate(xd, wd, H, V, 1e-6, dtype, gate_first=True, **kw).reshape(T, H, V), unit(X * s) * W, eps)


# columns within a warp's pieces, whole, a piece over, and behind 2,048; rows an expert beyond those taken together
@pytest.mark.parametrize("K,F", [(8, 8), (264, 72), (2048, 104), (2056, 24), (4104, 2056)])
@pytest.mark.parametrize("T", [1, 7, 11])
def test_few_rows_an_expert(K, F, T):
    from gopherllm_b200 import ops as o
    g = torch.Generator().manual_seed(K + T)
    E, top = 12, 2
    x = torch.randn(T, K, generator=g).bfloat16()
    wgu = (torch.randn(E, 2 * F, K, generator=g) * K ** -0.5).bfloat16()
    wd = (torch.randn(E, 16, F, generator=g) * F ** -0.5).bfloat16()
    ids = torch.rand(T, E, generator=g).argsort(-1)[:, :top].int()
    ids[:, 0] = 3                                    # one expert meets every token
    ids[:, 1] = torch.where(ids[:, 1] == 3, 4, ids[:, 1])
    wts = torch.rand(T, top, generator=g)
    got = o.moe_experts(x.cuda(), ids.cuda(), wts.cuda(), wgu.cuda(), wd.cuda())
    want = torch.zeros(T, 16, dtype=torch.float64)
    for t in range(T):
        for k in range(top):
            e = int(ids[t, k])
            y = wgu[e].double() @ x[t].double()
            h = (y[:F] * torch.sigmoid(y[:F]) * y[F:]).bfloat16().double()
            want[t] += wts[t, k].double() * (wd[e].double() @ h)
    # h is rounded to bfloat16 on both sides, from sums that differ in the last places: a unit of 2^-8 of an element, F of them
    close(got, want, 2 ** -7)
