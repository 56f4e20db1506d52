"""The selective scan's walks over chunks, a thread a channel: states of one to sixteen numbers, channels that leave a block part
empty, chunks and stages that end anywhere, against the recurrence in 64 bits."""
from types import SimpleNamespace

import pytest
import torch

from test_vopedra_gpu import check_selective_scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens", [1, 30, 64, 100])
@pytest.mark.parametrize("C,N", [(1, 16), (130, 5), (128, 1), (257, 12)])
def test_chunks_of_any_length(C, N, tokens, dtype, monkeypatch):
    from gopherllm_b200 import ops
    monkeypatch.setattr(ops, "scan_chunk_tokens", lambda *a: tokens)
    monkeypatch.setattr(ops, "scan_by_channel", lambda *a: True)
    check_selective_scan(C, N, [64, 1, 131, 65], dtype)


def test_endless_and_harsh_steps_in_chunks(monkeypatch):
    """An infinite step forgets the state and writes infinity from its token on, in its channel alone; steps so large that a
    state is gone at once leave what is left exact."""
    from gopherllm_b200 import ops
    monkeypatch.setattr(ops, "scan_chunk_tokens", lambda *a: 32)
    monkeypatch.setattr(ops, "scan_by_channel", lambda *a: True)
    C, N, T = 40, 16, 100
    g = torch.Generator().manual_seed(2)
    up = lambda *s: torch.rand(*s, generator=g) + 0.1  # noqa: E731
    x, bc, z, dtp, a_log, d_skip, state = up(T, C), up(T, 2 * N), up(T, C), 100.0 * up(T, C), up(C, N), up(C), up(1, C * N)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    ctx = SimpleNamespace(seq_slot=i32([0]), seq_qstart=i32([0]), seq_qlen=i32([T]), n_seqs=1, max_qlen=T, n_tokens=T)
    run = lambda d: ops.selective_scan(x.cuda(), d.cuda(), bc.cuda(), z.cuda(), 0, a_log.cuda(), d_skip.cuda(), state.cuda(), ctx).cpu()  # noqa: E731
    got = run(dtp).double()
    dt, S = dtp.double(), state.double().view(C, N)          # (softplus of numbers above 20 is the number)
    for t in range(T):
        step = torch.nn.functional.softplus(dt[t])
        S = torch.exp(-step[:, None] * torch.exp(a_log.double())) * S + (step * x[t].double())[:, None] * bc[t, :N].double()
        want = (S @ bc[t, N:].double() + d_skip.double() * x[t].double()) * torch.nn.functional.silu(z[t].double())
        assert ((got[t] - want).abs() <= 2e-5 * want.abs().max()).all(), t
    ended = dtp / 100.0
    ended[45, ::3] = float("inf")
    got = run(ended)
    assert torch.isfinite(got[:45]).all() and torch.isfinite(got[:, 1::3]).all() and (got[45:, ::3] == float("inf")).all()


def scan_call(C, N, T, seed=2):
    """Positive inputs of one run, and the call with some of them replaced."""
    from gopherllm_b200 import ops
    g = torch.Generator().manual_seed(seed)
    up = lambda *s: torch.rand(*s, generator=g) + 0.1  # noqa: E731
    inputs = dict(x=up(T, C), bc=up(T, 2 * N), z=up(T, C), dtp=up(T, C), a_log=up(C, N) - 1.0, d_skip=up(C))
    state = up(1, C * N)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    ctx = SimpleNamespace(seq_slot=i32([0]), seq_qstart=i32([0]), seq_qlen=i32([T]), n_seqs=1, max_qlen=T, n_tokens=T)

    def run(**other):
        t = {k: v.cuda() for k, v in {**inputs, **other}.items()}
        kept = state.cuda()
        out = ops.selective_scan(t["x"], t["dtp"], t["bc"], t["z"], 0, t["a_log"], t["d_skip"], kept, ctx)
        return out.cpu(), kept.cpu()
    return inputs, run


# states that fill the registers and that leave some of them unused
@pytest.mark.parametrize("N", [16, 13, 12, 5, 1])
def test_endless_steps_and_inputs_in_states_of_any_size(N, monkeypatch):
    """An infinite step, and an infinite input, write infinity from their token on in their channel alone."""
    from gopherllm_b200 import ops
    monkeypatch.setattr(ops, "scan_chunk_tokens", lambda *a: 32)
    monkeypatch.setattr(ops, "scan_by_channel", lambda *a: True)
    C, T, at = 40, 100, 45
    inputs, run = scan_call(C, N, T)
    whole, _ = run()
    for name in ("dtp", "x"):
        t = inputs[name].clone()
        t[at, ::3] = float("inf")
        got, kept = run(**{name: t})
        assert torch.equal(got[:at], whole[:at]) and torch.equal(got[:, 1::3], whole[:, 1::3]), name
        assert (got[at:, ::3] == float("inf")).all() and (kept.view(C, N)[::3] == float("inf")).all(), name


@pytest.mark.parametrize("N", [16, 5])
def test_a_decay_that_is_no_number(N, monkeypatch):
    """A rate that is NaN, and an infinite one at a step of zero: the channel is NaN from there on, as in the walk in one piece."""
    from gopherllm_b200 import ops
    C, T, at = 40, 100, 45
    inputs, run = scan_call(C, N, T)
    rate, step = inputs["a_log"].clone(), inputs["dtp"].clone()
    rate[3, N // 2], rate[7, N - 1] = float("nan"), float("inf")
    step[at, 7] = -200.0                              # (softplus of it is zero)
    monkeypatch.setattr(ops, "scan_by_channel", lambda *a: True)
    both = []
    for tokens in (0, 32):
        monkeypatch.setattr(ops, "scan_chunk_tokens", lambda *a: tokens)
        both.append(run(a_log=rate, dtp=step))
    for piece, chunks in zip(*both):
        assert torch.equal(piece.isnan(), chunks.isnan())
        assert torch.allclose(piece, chunks, rtol=1e-5, atol=1e-6, equal_nan=True)
    out = both[1][0]
    assert out[:, 3].isnan().all() and out[at:, 7].isnan().all() and torch.isfinite(out[:at, 7]).all()
    assert torch.isfinite(out[:, [c for c in range(C) if c not in (3, 7)]]).all()
