"""Which selective scans are walked in chunks, of how many tokens, and by which walk."""


def test_rule():
    from gopherllm_b200 import ops
    assert ops.scan_by_channel(64, 16, False) and ops.scan_by_channel(64, 9, False) and ops.scan_by_channel(1024, 16, True)
    for no in ((4096, 8, False), (4096, 17, False), (1023, 16, True), (4096, 1, True)):
        assert not ops.scan_by_channel(*no), no
    # in 32 bits, and where lanes share a channel: the longest run alone
    for C, N, exact in ((4096, 16, True), (64, 16, True), (4096, 8, False), (2048, 40, False)):
        for seqs in (1, 64):
            for longest in (1, 300, 1023, 1024, 5000):
                assert ops.scan_chunk_tokens(C, N, exact, seqs, seqs * longest, longest) == (128 if longest >= 1024 else 0)
    tokens = lambda C, qlens: ops.scan_chunk_tokens(C, 16, False, len(qlens), sum(qlens), max(qlens))  # noqa: E731
    assert tokens(4096, [255]) == 0 and tokens(4096, [256]) == 32 and tokens(4096, [1000]) == 32 and tokens(4096, [1100]) == 64
    assert tokens(512, [2040]) == 32 and tokens(1024, [300] * 16) == 64
    # single tokens beside a run: a chunk each
    assert tokens(4096, [300] + [1] * 63) == 0 and tokens(4096, [500] + [1] * 63) == 32 and tokens(1024, [300] + [1] * 63) == 32
    # every (sequence, chunk) keeps a whole state
    assert tokens(4096, [8192] * 64) == 128
