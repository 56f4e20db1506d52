"""The scalar-decay memories' chunks as products on the tensor cores, against the recurrence in 64 bits."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def make(kind, H, D, V, KVH, half, qlens, seed, ld_more=0, fixed=False, harsh=False):
    """Inputs of a call in bfloat16, and the call (with ``ld_more`` = 1 the rows begin anywhere, which the products do not take)."""
    from gopherllm_b200 import ops
    g = torch.Generator().manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    B, T = len(qlens), sum(qlens)
    cols = 2 * KVH * D + H * V + 2 * H
    proj = rn(T, -(-cols // 8) * 8 + ld_more).bfloat16()
    a_log, dt_bias, skip = rn(H) * 0.7, rn(H) + (3.0 if harsh else -3.0), rn(H)
    decay = torch.rand(H, generator=g) ** 0.1
    if harsh:
        decay[0], a_log[-1] = 0.0, 4.0                        # forgets everything at every token
    angle = torch.rand(T, max(1, half), generator=g) * 6.28
    state = rn(B + 1, ops.memory_state_size(kind, H, D, V)) * 0.3
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    ctx = SimpleNamespace(seq_slot=i32(list(range(1, B + 1))), seq_qstart=i32([sum(qlens[:i]) for i in range(B)]), seq_qlen=i32(qlens),
                          tok_seq=i32([b for b in range(B) for _ in range(qlens[b])]), n_seqs=B, max_qlen=max(qlens), n_tokens=T)
    KD, off = KVH * D, 2 * KVH * D + H * V
    scale = dict(q_scale=D ** -0.5, k_scale=0.7) if kind == 3 else dict(q_scale=D ** -0.5)

    def call(proj=proj):
        kept, p = state.cuda(), proj.cuda()
        if kind == 0:
            out = ops.memory_scan(0, p, kept, ctx, H, D, V, 0, KD, 2 * KD, off, off + H, cap=15.0, **scale)
        else:
            gates = {} if fixed else dict(gates=p, a_log=a_log.cuda(), dt_bias=dt_bias.cuda())
            turn = dict(cos=torch.cos(angle).cuda(), sin=torch.sin(angle).cuda()) if half else {}
            out = ops.memory_scan(3, p, kept, ctx, H, D, V, 0, KD, 2 * KD, 0, off, kv_heads=KVH, decay=decay.cuda() if fixed else None,
                                  skip=skip.cuda(), **gates, **turn, **scale)
        return out.cpu(), kept.cpu()

    def exact():
        p = proj.double()
        q, k = (p[:, i * KD:(i + 1) * KD].view(T, KVH, D).clone() for i in (0, 1))
        if half:
            c, s = torch.cos(angle).double()[:, None], torch.sin(angle).double()[:, None]
            q, k = (torch.cat([x[..., :half] * c - x[..., half:2 * half] * s, x[..., half:2 * half] * c + x[..., :half] * s,
                               x[..., 2 * half:]], -1) for x in (q, k))
        q, k = (x.repeat_interleave(H // KVH, 1) for x in (q, k))
        q, k = q * scale["q_scale"], k * scale.get("k_scale", 1.0)
        v, gates = p[:, 2 * KD:off].view(T, H, V), p[:, off:]
        rows, out, t = state.double().clone(), torch.empty(T, H, V, dtype=torch.float64), 0
        for b, n in enumerate(qlens):
            row, HD = rows[b + 1], H * D
            S = row[:HD * V].view(H, D, V).clone()
            if kind == 0:
                norm, m = row[HD * V:HD * V + HD].view(H, D).clone(), row[HD * V + HD:HD * V + HD + H].clone()
            for _ in range(n):
                if kind == 0:
                    gi, gf = 15.0 * torch.tanh(gates[t, :H] / 15.0), torch.nn.functional.logsigmoid(15.0 * torch.tanh(gates[t, H:2 * H] / 15.0))
                    m2 = torch.maximum(gf + m, gi)
                    keep, take, m = torch.exp(gf + m - m2), torch.exp(gi - m2), m2
                    norm = keep[:, None] * norm + take[:, None] * k[t]
                elif fixed:
                    keep, take = decay.double(), torch.ones(H, dtype=torch.float64)
                else:
                    take = torch.nn.functional.softplus(gates[t, :H] + dt_bias.double())
                    keep = torch.exp(-torch.exp(a_log.double()) * take)
                S = keep[:, None, None] * S + (take[:, None] * k[t])[:, :, None] * v[t][:, None, :]
                y = torch.einsum("hdv,hd->hv", S, q[t])
                if kind == 0:
                    y = y / (torch.maximum((norm * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
                else:
                    y = y + skip.double()[:, None] * v[t]
                out[t] = y
                t += 1
            row[:HD * V] = S.reshape(-1)
            if kind == 0:
                row[HD * V:HD * V + HD], row[HD * V + HD:] = norm.reshape(-1), m
        return out.reshape(T, H * V), rows

    return proj, call, exact


# columns that fill a block and that do not; turned dims none, some and all; heads that share keys; runs that end at a chunk's edges
SIZES = [(0, 2, 64, 64, 2, 0), (0, 2, 128, 72, 2, 0), (3, 4, 128, 64, 2, 0), (3, 4, 64, 136, 4, 32), (3, 2, 64, 8, 1, 8), (3, 2, 128, 64, 2, 64)]


@pytest.mark.parametrize("chunk", [32, 64])
@pytest.mark.parametrize("fixed,harsh", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("kind,H,D,V,KVH,half", SIZES)
def test_products_and_the_walk(kind, H, D, V, KVH, half, fixed, harsh, chunk, monkeypatch):
    from gopherllm_b200 import ops
    if kind == 0 and (fixed or harsh):
        pytest.skip("the gated kind has gates of its own")
    monkeypatch.setattr(ops, "memory_chunk_tokens", lambda *a: chunk)
    launches, check = [], ops._check
    monkeypatch.setattr(ops, "_check", lambda code, what, kernels=1: (launches.append(kernels), check(code, what, kernels)))
    qlens = [1, 17, 63, 64, 65, 200]
    errors = {}
    for more, form in ((0, "products"), (1, "walk")):            # (rows that begin anywhere are walked)
        proj, call, exact = make(kind, H, D, V, KVH, half, qlens, H + D + V, ld_more=more, fixed=fixed, harsh=harsh)
        assert ops.memory_takes_products(kind, proj.dtype, proj.shape[1], D, V, (0, KVH * D, 2 * KVH * D), half) == (form == "products")
        launches.clear()
        both = call()
        assert launches == [(2 if kind == 0 else 1) + (3 if form == "products" else 5 if kind == 0 else 4)], (form, launches)
        for got, ref, what in zip(both, exact(), ("results", "states")):
            # a few roundings of 2^-24 of the largest partial sum a token, and of its decays
            bound = 2 ** -22 * max(qlens) * max(1.0, float(ref.abs().max()))
            err = float((got.double() - ref).abs().max())
            assert err <= bound, (form, what, err, bound)
            errors[form, what] = float((got.double() - ref).norm() / ref.norm())
    # factors of 24 bits: no further from 64-bit than the walk, but for roundings that fall the other way; factors of two bfloat16
    # parts, 16 bits, would be off by some 2^-18 each
    for what in ("results", "states"):
        assert errors["products", what] <= min(2.0 * errors["walk", what] + 2 ** -24, 1e-6), errors


@pytest.mark.parametrize("kind,H,D,V,KVH,half", SIZES)
def test_a_value_that_is_no_number_stays_behind_its_token(kind, H, D, V, KVH, half, monkeypatch):
    """An infinite or NaN value shows in its column from its token on, in its sequence alone, and nowhere else."""
    from gopherllm_b200 import ops
    monkeypatch.setattr(ops, "memory_chunk_tokens", lambda *a: 64)
    qlens = [70, 130, 64]
    proj, call, _ = make(kind, H, D, V, KVH, half, qlens, 3)
    whole, rows = call()
    at = qlens[0] + 75                                       # in the second sequence's second chunk
    for bad, col in ((float("inf"), 5), (float("-inf"), V - 1), (float("nan"), 0)):
        p = proj.clone()
        p[at, 2 * KVH * D + V + col] = bad                   # head 1
        got, kept = call(p)
        hit = torch.zeros_like(got, dtype=torch.bool)
        hit[at:qlens[0] + qlens[1], V + col] = True
        assert not torch.isfinite(got[hit]).any() and torch.equal(got[~hit], whole[~hit])
        S, S0 = (r[:, :H * D * V].view(-1, H, D, V) for r in (kept, rows))
        lost = torch.zeros_like(S, dtype=torch.bool)
        lost[2, 1, :, col] = True
        assert not torch.isfinite(S[lost]).any() and torch.equal(S[~lost], S0[~lost])


@pytest.mark.parametrize("what", ["gate", "second gate", "key", "query"])
@pytest.mark.parametrize("place", [74, 75])                  # an even and an odd place of a chunk: a lane holds two tokens' gates
@pytest.mark.parametrize("kind,H,D,V,KVH,half", SIZES)
def test_a_gate_or_key_that_is_no_number_stays_behind_its_token(kind, H, D, V, KVH, half, place, what, monkeypatch):
    """A NaN in a gate or a key shows in its heads' rows from its token on, one in a query in its own row, in its sequence alone; every
    other row is the same bit for bit."""
    from gopherllm_b200 import ops
    if kind == 3 and what == "second gate":
        pytest.skip("the plain decay has one gate")
    monkeypatch.setattr(ops, "memory_chunk_tokens", lambda *a: 64)
    qlens = [70, 130, 64]
    proj, call, _ = make(kind, H, D, V, KVH, half, qlens, 5)
    whole, _ = call()
    at, end, KD, off = qlens[0] + place, qlens[0] + qlens[1], KVH * D, 2 * KVH * D + H * V
    heads = [H - 1] if "gate" in what else list(range((KVH - 1) * (H // KVH), H))
    p = proj.clone()
    p[at, {"gate": off + H - 1, "second gate": off + 2 * H - 1, "key": 2 * KD - 1, "query": KD - 1}[what]] = float("nan")
    got, _ = call(p)
    hit = torch.zeros(sum(qlens), H, V, dtype=torch.bool)
    for h in heads:
        hit[at:at + 1 if what == "query" else end, h] = True
    hit = hit.view(sum(qlens), H * V)
    assert not torch.isfinite(got[hit]).any() and torch.equal(got[~hit], whole[~hit])
