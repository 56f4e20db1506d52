"""The Vopedra design through the library's loader, cache, step function, scheduler and kernels,
against the plain implementation (tests/plain_vopedra.py) on small models whose weights the tests
make themselves."""
import numpy as np
import pytest
import torch

import plain_vopedra as pv
import vopedra_models as vm

pytestmark = pytest.mark.gpu

# the largest |difference| of a position's logits is bounded by TOL * max(1, max|reference|); in bfloat16
# (small widths, unit-gain random weights, up to seven layer runs) also the mean over positions by MEAN_TOL
TOL = {"float32": 3e-4, "bfloat16": 1e-1}
MEAN_TOL = {"float32": 1e-4, "bfloat16": 3e-2}
_REF = {}


def plain_logits(folder, tokens):
    key = (folder, tuple(tokens))
    if key not in _REF:
        cfg, t = pv.read_folder(folder)
        _REF[key] = pv.forward(cfg, t, list(tokens)).numpy()
    return _REF[key]


def load(folder, dtype, max_tokens=4096, **kw):
    import gopherllm_b200 as gl
    return gl.load(folder, dtype=dtype, max_tokens=max_tokens, **kw)


def feed(model, slot, tokens, cuts):
    """Feed ``tokens`` in pieces of the given sizes (the rest one by one); logits of every position."""
    out, at = [], 0
    cuts = list(cuts)
    while at < len(tokens):
        n = min(cuts.pop(0) if cuts else 1, len(tokens) - at)
        out.append(model.step([(slot, tokens[at:at + n])], [list(range(n))]).cpu().numpy())
        at += n
    return np.concatenate(out, 0)


def check(got, ref, dtype, what=""):
    assert got.shape == ref.shape, (got.shape, ref.shape)
    assert np.isfinite(got).all(), what
    err = np.abs(got - ref).max(-1)
    bound = TOL[dtype] * max(1.0, float(np.abs(ref).max()))
    worst = int(err.argmax())
    assert err.max() <= bound, f"{what} {dtype}: position {worst} differs by {err.max():.3e} (bound {bound:.3e})"
    mean_bound = MEAN_TOL[dtype] * max(1.0, float(np.abs(ref).max()))
    assert err.mean() <= mean_bound, f"{what} {dtype}: positions differ by {err.mean():.3e} on average (bound {mean_bound:.3e})"


def tokens_for(cfg, n, seed):
    return [int(t) for t in np.random.default_rng(seed).integers(0, cfg["vocab"], size=n)]


FOLDERS = {}


def folder_for(name, cfg, seed, **kw):
    key = (name, seed, tuple(sorted(kw.items())))
    if key not in FOLDERS:
        FOLDERS[key] = vm.write_folder(cfg, vm.draw(cfg, seed, **kw))
    return FOLDERS[key]


ALONE = [("mlstm", vm.only(vm.ALPHA, 0)), ("mlstm_bare_wide", vm.only(vm.BETA, 2, mlp=False)),
         ("mamba1", vm.only(vm.ALPHA, 1)), ("mamba1_short_filter", vm.only(vm.BETA, 1)), ("mamba1_one_tap", vm.only(vm.GAMMA, 0)),
         ("pair", vm.only(vm.ALPHA, 2)), ("pair_full_rotation", vm.only(vm.BETA, 0, mlp=False)),
         ("pair_no_rotation", vm.only(vm.GAMMA, 1)),
         ("pair_looped", vm.only(vm.ALPHA, 2, loop={"start": 0, "stop": 1, "times": 2}))]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name,cfg", ALONE, ids=[a[0] for a in ALONE])
def test_each_mechanism_alone(name, cfg, dtype):
    """One layer of one kind: a whole prompt across a page's edge, then single tokens."""
    folder = folder_for(name, cfg, 11)
    toks = tokens_for(cfg, 78, 1)
    m = load(folder, dtype)
    s = m.open_sequence()
    got = feed(m, s, toks, [70])
    m.engine.check_device()
    check(got, plain_logits(folder, toks), dtype, name)
    m.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("cfg_name", ["ALPHA", "BETA", "GAMMA", "DELTA"])
def test_whole_pieces_and_single_tokens(cfg_name, dtype):
    """The same tokens whole, in pieces of many sizes down to two, and mostly one by one."""
    cfg = getattr(vm, cfg_name)
    folder = folder_for(cfg_name, cfg, 5)
    toks = tokens_for(cfg, 150, 2)
    ref = plain_logits(folder, toks)
    m = load(folder, dtype)
    for cuts in ([150], [2, 2, 3, 57, 1, 64, 2, 19], [40]):
        s = m.open_sequence()
        got = feed(m, s, toks, cuts)
        m.close_sequence(s)
        check(got, ref, dtype, f"{cfg_name} cuts {cuts}")
    m.engine.check_device()
    m.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_first_tokens(dtype):
    folder = folder_for("ALPHA", vm.ALPHA, 5)
    m = load(folder, dtype)
    for n in (1, 2, 3):
        toks = tokens_for(vm.ALPHA, n, 20 + n)
        s = m.open_sequence()
        check(feed(m, s, toks, [n]), plain_logits(folder, toks), dtype, f"{n} tokens")
        m.close_sequence(s)
    m.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_unequal_batch_against_each_alone(dtype):
    """Three prompts of different lengths as one batch, then decoded together while the shorter ones
    leave; every sequence must get what it gets alone."""
    cfg = vm.ALPHA
    folder = folder_for("ALPHA", cfg, 5)
    lens, prompt = [9, 140, 71], [5, 131, 66]
    seqs = [tokens_for(cfg, n, 30 + i) for i, n in enumerate(lens)]
    m = load(folder, dtype)
    slots = [m.open_sequence() for _ in seqs]
    got = [[] for _ in seqs]
    out = m.step([(slots[i], seqs[i][:prompt[i]]) for i in range(3)], [list(range(p)) for p in prompt]).cpu().numpy()
    at = 0
    for i, p in enumerate(prompt):
        got[i].append(out[at:at + p])
        at += p
    pos = list(prompt)
    while any(pos[i] < lens[i] for i in range(3)):
        live = [i for i in range(3) if pos[i] < lens[i]]
        out = m.step([(slots[i], [seqs[i][pos[i]]]) for i in live]).cpu().numpy()
        for r, i in enumerate(live):
            got[i].append(out[r:r + 1])
            pos[i] += 1
            if pos[i] == lens[i]:
                m.close_sequence(slots[i])
    m.engine.check_device()
    for i in range(3):
        check(np.concatenate(got[i], 0), plain_logits(folder, seqs[i]), dtype, f"sequence {i} in the batch")
    if dtype == "float32":
        alone = load(folder, dtype)
        s = alone.open_sequence()
        one = feed(alone, s, seqs[2], [prompt[2]])
        assert np.abs(one - np.concatenate(got[2], 0)).max() <= 2e-5 * max(1.0, np.abs(one).max())
        alone.close()
    m.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_slots_and_pages_used_again(dtype):
    """A sequence that takes the slot, the state rows and the pages another one left must not see them."""
    cfg = vm.ALPHA
    folder = folder_for("ALPHA", cfg, 5, long_memory=True)
    a, b, c = tokens_for(cfg, 130, 40), tokens_for(cfg, 90, 41), tokens_for(cfg, 70, 42)
    m = load(folder, dtype, max_tokens=512)
    sa = m.open_sequence()
    feed(m, sa, a, [100])
    sb = m.open_sequence()
    gb = [feed(m, sb, b[:50], [50])]
    m.close_sequence(sa)
    sc = m.open_sequence()                      # takes a's slot and pages while b is still live
    assert sc == sa
    gc = feed(m, sc, c, [33, 2])
    gb.append(feed(m, sb, b[50:], [7]))
    m.engine.check_device()
    check(gc, plain_logits(folder, c), dtype, "the sequence in the used slot")
    check(np.concatenate(gb, 0), plain_logits(folder, b), dtype, "the sequence that stayed")
    m.engine.cache.check()
    m.close()


def test_far_tokens_and_page_edges():
    """Weights with long memories and a sharp softmax: the logits late in a sequence hang on single
    tokens hundreds of positions back and on keys right at the pages' edges."""
    cfg = vm.ALPHA
    folder = folder_for("ALPHA_far", cfg, 7, long_memory=True, sharp=4.0)
    toks = tokens_for(cfg, 200, 50)
    ref = plain_logits(folder, toks)
    other = list(toks)
    other[3] = (other[3] + 1) % cfg["vocab"]
    moved = np.abs(plain_logits(folder, other)[190:] - ref[190:]).max()
    assert moved > 20 * TOL["float32"] * max(1.0, np.abs(ref).max()), "the test's model forgets its early tokens"
    m = load(folder, "float32")
    for cuts in ([200], [63, 1, 1, 63, 2], [129], [64, 64, 64]):
        s = m.open_sequence()
        check(feed(m, s, toks, cuts), ref, "float32", f"cuts {cuts}")
        m.close_sequence(s)
    m.close()
    m = load(folder, "bfloat16")
    s = m.open_sequence()
    got = feed(m, s, toks, [127])
    m.engine.check_device()
    check(got, ref, "bfloat16", "far tokens")
    m.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_long_decoding(dtype):
    """A few tokens of prompt, then single tokens across two pages' edges (captured steps in bfloat16)."""
    cfg = vm.BETA
    folder = folder_for("BETA", cfg, 9, long_memory=True)
    toks = tokens_for(cfg, 140, 60)
    m = load(folder, dtype)
    s = m.open_sequence()
    got = feed(m, s, toks, [3])
    m.engine.check_device()
    check(got, plain_logits(folder, toks), dtype, "long decoding")
    m.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_long_runs_walked_as_chunks(dtype, monkeypatch):
    """Long runs of the scans are cut into chunks that are walked side by side, with a carry between two
    walks.  With chunks of 16 tokens from 32 tokens on: a whole prompt (a ragged last chunk), pieces above
    and below the threshold, and a batch whose shorter sequence has fewer chunks than the longer one."""
    from gopherllm_b200 import ops
    monkeypatch.setattr(ops, "SCAN_CHUNK_TOKENS", 16)
    monkeypatch.setattr(ops, "SCAN_CHUNKED_FROM", 32)
    monkeypatch.setattr(ops, "SCAN_SHORT_CHUNKED_FROM", 32)             # (states of more than 8 numbers in bfloat16 have lines of their own)
    monkeypatch.setattr(ops, "SCAN_SHORT_CHUNK_TOKENS", 16)
    monkeypatch.setattr(ops, "SCAN_SHORT_CHUNK_TOKENS_FEW", 16)
    for cfg_name in ("ALPHA", "BETA"):
        cfg = getattr(vm, cfg_name)
        folder = folder_for(cfg_name, cfg, 5, long_memory=True)
        toks = tokens_for(cfg, 150, 2)
        ref = plain_logits(folder, toks)
        m = load(folder, dtype)
        for cuts in ([150], [33, 31, 64, 17]):
            s = m.open_sequence()
            check(feed(m, s, toks, cuts), ref, dtype, f"{cfg_name} cuts {cuts}")
            m.close_sequence(s)
        short = tokens_for(cfg, 37, 3)
        sa, sb = m.open_sequence(), m.open_sequence()
        out = m.step([(sa, short), (sb, toks[:100])], [list(range(37)), list(range(100))]).cpu().numpy()
        check(out[:37], plain_logits(folder, short), dtype, "the shorter of two")
        check(out[37:], ref[:100], dtype, "the longer of two")
        m.engine.check_device()
        m.close()


def test_greedy_generation_through_the_scheduler():
    """Model.generate, greedy, for prompts of different lengths in one call: the tokens the plain
    implementation chooses."""
    cfg = vm.GAMMA
    folder = folder_for("GAMMA", cfg, 3)
    prompts = [tokens_for(cfg, n, 70 + n) for n in (4, 37, 66)]
    m = load(folder, "float32")
    outs = m.generate(prompts, max_tokens=8, temperature=0.0, top_k=0, top_p=1.0, repeat_penalty=1.0, stop_tokens=())
    pcfg, t = pv.read_folder(folder)
    for p, o in zip(prompts, outs):
        seq = list(p)
        for _ in range(8):
            logits = pv.forward(pcfg, t, seq)[-1]
            top2 = torch.topk(logits, 2).values
            if float(top2[0] - top2[1]) < 1e-3:        # a tie within rounding proves nothing either way
                break
            seq.append(int(logits.argmax()))
        want = seq[len(p):]
        assert o.tokens[:len(want)] == want, (o.tokens, want)
    m.close()
    mb = load(folder, "bfloat16")
    outs_b = mb.generate(prompts, max_tokens=8, temperature=0.0, top_k=0, top_p=1.0, repeat_penalty=1.0, stop_tokens=())
    assert all(len(o.tokens) == 8 for o in outs_b)
    mb.engine.check_device()
    mb.close()


def test_replay_of_a_trace(tmp_path):
    """The trace runner's loop on a Vopedra model: a batch of two requests, one ends, the other goes on."""
    import json
    from gopherllm_b200.engine.replay import run
    cfg = vm.ALPHA
    folder = folder_for("ALPHA", cfg, 5)
    a, b = tokens_for(cfg, 70, 80), tokens_for(cfg, 12, 81)
    lines = [json.dumps({"step": 0, "entries": [{"id": "a", "tokens": a[:66], "want": [0, 63, 65]},
                                                 {"id": "b", "tokens": b[:11], "want": []}], "end": []}),
             json.dumps({"step": 1, "entries": [{"id": "a", "tokens": a[66:67], "want": [0]},
                                                 {"id": "b", "tokens": b[11:], "want": [0]}], "end": ["b"]})]
    lines += [json.dumps({"step": 2 + i, "entries": [{"id": "a", "tokens": [a[67 + i]], "want": [0]}],
                          "end": ["a"] if i == 2 else []}) for i in range(3)]
    m = load(folder, "float32")
    said = []
    run(m, lines, str(tmp_path), said.append)
    assert said == [f"done {i}" for i in range(5)]
    ra, rb = plain_logits(folder, a), plain_logits(folder, b)
    got0 = np.fromfile(tmp_path / "0.f32", dtype="<f4").reshape(3, -1)
    check(got0, ra[[0, 63, 65]], "float32", "step 0")
    got1 = np.fromfile(tmp_path / "1.f32", dtype="<f4").reshape(2, -1)
    check(got1, np.stack([ra[66], rb[11]]), "float32", "step 1")
    got4 = np.fromfile(tmp_path / "4.f32", dtype="<f4").reshape(1, -1)
    check(got4, ra[69:70], "float32", "step 4")
    assert not m.engine.cache.live_slots()
    m.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C,N,qlens", [(40, 16, [1, 1, 1]), (40, 16, [1, 2, 3, 4, 5, 15]), (24, 4, [16, 17, 33]), (72, 24, [31, 6]),
                                       (16, 40, [20, 1]), (3000, 16, [5, 40] * 8)])
def test_selective_scan_forms(C, N, qlens, dtype):
    """Runs that end inside a group of tokens and inside a staged chunk, one token a sequence, states of fewer lanes than a
    group, of no power of two and too many to fetch ahead, and many sequences, against the recurrence in 64-bit."""
    check_selective_scan(C, N, qlens, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens", [48, 128])
@pytest.mark.parametrize("C,N,qlens", [(40, 16, [50, 129, 300, 1]), (24, 40, [300, 50, 129]), (3000, 16, [128, 257])])
def test_selective_scan_in_chunks_of_several_stages(C, N, qlens, tokens, dtype, monkeypatch):
    """Chunks as long as those of long prompts, so that inputs fetched ahead cross a chunk's stages: ragged last stages and last
    chunks, runs of one chunk and of many, states that are fetched ahead and states that are not."""
    from gopherllm_b200 import ops
    monkeypatch.setattr(ops, "SCAN_CHUNKED_FROM", 64)
    monkeypatch.setattr(ops, "SCAN_CHUNK_TOKENS", tokens)
    monkeypatch.setattr(ops, "SCAN_SHORT_CHUNKED_FROM", 64)
    monkeypatch.setattr(ops, "SCAN_SHORT_CHUNK_TOKENS", tokens)
    monkeypatch.setattr(ops, "SCAN_SHORT_CHUNK_TOKENS_FEW", tokens)
    monkeypatch.setattr(ops, "SCAN_SHORT_STATES", 1 << 30)
    assert ops.scan_chunk_tokens(C, N, dtype == torch.float32, len(qlens), sum(qlens), max(qlens)) == tokens
    for by_channel in (False, True) if N <= ops.SCAN_CHANNEL_STATE else (False,):       # both walks over chunks, whichever these sizes take
        monkeypatch.setattr(ops, "scan_by_channel", lambda *a: by_channel)
        check_selective_scan(C, N, qlens, dtype)


def check_selective_scan(C, N, qlens, dtype):
    from types import SimpleNamespace
    from gopherllm_b200 import ops
    g = torch.Generator().manual_seed(C + N)
    T, B, dev = sum(qlens), len(qlens), "cuda:0"
    rn = lambda *s: torch.randn(*s, generator=g)
    x, bc, z = rn(T, C).to(dtype), rn(T, 2 * N).to(dtype), rn(T, C + 8).to(dtype)
    dtp, a_log, d_skip, state = rn(T, C) - 3, rn(C, N), rn(C), rn(B + 1, C * N)
    starts = [sum(qlens[:i]) for i in range(B)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    ctx = SimpleNamespace(seq_slot=i32(list(range(1, B + 1))), seq_qstart=i32(starts), seq_qlen=i32(qlens), n_seqs=B, max_qlen=max(qlens), n_tokens=T)
    kept = state.to(dev)
    got = ops.selective_scan(x.to(dev), dtp.to(dev), bc.to(dev), z.to(dev), 8, a_log.to(dev), d_skip.to(dev), kept, ctx).cpu().double()
    xd, bd, zd = x.double(), bc.double(), z.double()[:, 8:]
    dt, A = torch.nn.functional.softplus(dtp.double()), -torch.exp(a_log.double())
    want = torch.empty(T, C, dtype=torch.float64)
    for b in range(B):
        S = state[b + 1].double().view(C, N)
        for t in range(starts[b], starts[b] + qlens[b]):
            S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * xd[t])[:, None] * bd[t, :N]
            want[t] = (S @ bd[t, N:] + d_skip.double() * xd[t]) * torch.nn.functional.silu(zd[t])
        scale = max(1.0, S.abs().max().item())
        assert (kept[b + 1].cpu().double() - S.reshape(-1)).abs().max() <= 2e-6 * max(qlens) * scale      # 2^-22 a token
    tol = 2e-5 if dtype == torch.float32 else 2 ** -8
    assert (got - want).abs().max() <= tol * max(1.0, want.abs().max().item())
    assert torch.equal(kept[0].cpu(), state[0])


@pytest.mark.parametrize("N", [16, 24, 5])
@pytest.mark.parametrize("qlens", [[1, 1], [7, 20]])
def test_selective_scan_with_an_endless_step(N, qlens):
    """A step size that overflows to infinity forgets the state and writes infinity: nothing turns into NaN, also where the
    lanes that share a channel hold more places than it has states."""
    from types import SimpleNamespace
    from gopherllm_b200 import ops
    C, T, B, dev = 40, sum(qlens), len(qlens), "cuda:0"
    g = torch.Generator().manual_seed(N)
    up = lambda *s: torch.rand(*s, generator=g) + 0.1
    x, bc, z, dtp, a_log, d_skip, state = up(T, C), up(T, 2 * N), up(T, C), up(T, C), up(C, N), up(C), up(B, C * N)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    starts = [sum(qlens[:i]) for i in range(B)]
    for b, at in enumerate(starts):
        dtp[at + qlens[b] // 2, ::3] = float("inf")
    ctx = SimpleNamespace(seq_slot=i32(list(range(B))), seq_qstart=i32(starts), seq_qlen=i32(qlens), n_seqs=B, max_qlen=max(qlens), n_tokens=T)
    got = ops.selective_scan(x.to(dev), dtp.to(dev), bc.to(dev), z.to(dev), 0, a_log.to(dev), d_skip.to(dev), state.to(dev), ctx).cpu()
    for b, at in enumerate(starts):
        hit = at + qlens[b] // 2
        assert torch.isfinite(got[at:hit]).all() and torch.isfinite(got[at:at + qlens[b], 1::3]).all()
        assert (got[hit:at + qlens[b], ::3] == float("inf")).all()


def _memory_call(kind, H, D, V, qlens, dtype, seed, only=None):
    """A gated (0) or bounded-forget (1) memory's run: its inputs on the CPU, and the call on the GPU with a fresh copy of the
    states.  ``only``: the run of that sequence alone, with the inputs it has among the others."""
    from types import SimpleNamespace
    from gopherllm_b200 import ops
    g = torch.Generator().manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g)
    B, T, dev = len(qlens), sum(qlens), "cuda:0"
    pad = -(-2 * H // 8) * 8
    proj = rn(T, 2 * H * D + H * V + (pad if kind == 0 else 0)).to(dtype)
    lower = torch.rand(H * D, generator=g) * 0.9
    state = rn(B + 1, ops.memory_state_size(kind, H, D, V)) * 0.3
    if only is not None:
        at = sum(qlens[:only])
        proj, state, qlens = proj[at:at + qlens[only]], state[[0, only + 1]], [qlens[only]]
        B, T = 1, qlens[0]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    ctx = SimpleNamespace(seq_slot=i32(list(range(1, B + 1))), seq_qstart=i32([sum(qlens[:i]) for i in range(B)]), seq_qlen=i32(qlens),
                          tok_seq=i32([b for b in range(B) for _ in range(qlens[b])]), n_seqs=B, max_qlen=max(qlens), n_tokens=T)
    HD = H * D

    def call():
        kept, x = state.to(dev), proj.to(dev)
        if kind == 0:
            out = ops.memory_scan(0, x, kept, ctx, H, D, V, 0, HD, 2 * HD, 2 * HD + H * V, 2 * HD + H * V + H, cap=15.0, q_scale=D ** -0.5)
        else:
            out = ops.memory_scan(1, x, kept, ctx, H, D, V, 0, 0, 2 * HD, 0, HD, lower=lower.to(dev))
        return out.cpu(), kept.cpu()
    return proj, lower, state, call


def _memory_in_64_bits(kind, H, D, V, qlens, proj, lower, state):
    proj, HD = proj.double(), H * D
    q, v = proj[:, :HD].view(-1, H, D), proj[:, 2 * HD:2 * HD + H * V].view(-1, H, V)
    second = proj[:, HD:2 * HD].view(-1, H, D)
    out, rows, t = torch.empty(proj.shape[0], H, V, dtype=torch.float64), state.double().clone(), 0
    for b, n in enumerate(qlens):
        row = rows[b + 1]
        S = row[:HD * V].view(H, D, V).clone()
        if kind == 0:
            norm, m = row[HD * V:HD * V + HD].view(H, D).clone(), row[HD * V + HD:HD * V + HD + H].clone()
            gates = proj[:, 2 * HD + H * V:]
            gi = 15.0 * torch.tanh(gates[:, :H] / 15.0)
            gf = torch.nn.functional.logsigmoid(15.0 * torch.tanh(gates[:, H:2 * H] / 15.0))
        for _ in range(n):
            if kind == 0:
                m2 = torch.maximum(gf[t] + m, gi[t])
                keep, take, m = torch.exp(gf[t] + m - m2), torch.exp(gi[t] - m2), m2
                S = keep[:, None, None] * S + take[:, None, None] * second[t][:, :, None] * v[t][:, None, :]
                norm = keep[:, None] * norm + take[:, None] * second[t]
                qt = q[t] * D ** -0.5
                den = torch.maximum((norm * qt).sum(-1).abs(), torch.exp(-m)) + 1e-6
                out[t] = torch.einsum("hdv,hd->hv", S, qt) / den[:, None]
            else:
                low = lower.double().view(H, D)
                f = low + (1 - low) * torch.sigmoid(second[t])
                S = f[:, :, None] * S + (1 - f)[:, :, None] * v[t][:, None, :]
                out[t] = torch.einsum("hdv,hd->hv", S, torch.nn.functional.silu(q[t]))
            t += 1
        rows[b + 1, :HD * V] = S.reshape(-1)
        if kind == 0:
            rows[b + 1, HD * V:HD * V + HD], rows[b + 1, HD * V + HD:HD * V + HD + H] = norm.reshape(-1), m
    return out.reshape(-1, H * V), rows


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,D,V", [(2, 16, 32), (3, 24, 40), (2, 128, 64)])
@pytest.mark.parametrize("kind", [0, 1])
def test_memories_token_by_token_and_in_chunks(kind, H, D, V, dtype, monkeypatch):
    """The gated and the bounded-forget memory from states that are not zero, unequal runs beside one another (one token, whole
    chunks, ragged last ones), in both forms and with every length of chunk, against the recurrence in 64 bits.  The bound:
    a token adds a few roundings of 2^-24 to a sum and to the decays in front of it; a gated result is a quotient of two."""
    from gopherllm_b200 import ops
    qlens = [1, 33, 64, 129, 200]
    proj, lower, state, call = _memory_call(kind, H, D, V, qlens, dtype, 7 + D)
    want, rows = _memory_in_64_bits(kind, H, D, V, qlens, proj, lower, state)
    for chunk in (0, 32, 64, 128, 256):
        monkeypatch.setattr(ops, "memory_chunk_tokens", lambda *a: chunk)
        got, kept = call()
        for x, y, what in ((got, want, "results"), (kept, rows, "states")):
            bound = 2 ** -22 * max(qlens) * max(1.0, float(y.abs().max()))
            assert (x.double() - y).abs().max() <= bound, (what, chunk, float((x.double() - y).abs().max()), bound)
        assert torch.equal(kept[0], state[0])


@pytest.mark.parametrize("kind,H,D,V,n", [(0, 8, 128, 256, 300), (1, 32, 32, 64, 500), (0, 2, 16, 32, 1100)])
def test_32_bit_states_do_not_depend_on_how_many_run_beside(kind, H, D, V, n):
    """A prompt alone and among others of its length: the same state, bit for bit."""
    together = _memory_call(kind, H, D, V, [n] * 4, torch.float32, 5)[3]()[1]
    for b in range(4):
        alone = _memory_call(kind, H, D, V, [n] * 4, torch.float32, 5, only=b)[3]()[1]
        assert torch.equal(alone[1], together[b + 1]), b
