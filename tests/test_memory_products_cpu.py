"""Which memories' chunks are products on the tensor cores, and from how many tokens on."""
import torch


def test_rule():
    from gopherllm_b200 import ops
    takes = lambda kind=0, dtype=torch.bfloat16, ld=4096, D=128, V=256, offs=(0, 1024, 2048), half=0: ops.memory_takes_products(  # noqa: E731
        kind, dtype, ld, D, V, offs, half)
    assert takes() and takes(kind=3, D=64, V=8, half=32)
    for no in (dict(kind=1), dict(kind=2), dict(dtype=torch.float32), dict(D=32), dict(D=96), dict(V=60), dict(ld=4100), dict(offs=(0, 4, 8)), dict(half=12)):
        assert not takes(**no), no
    tokens = lambda n, seqs=1, **kw: ops.memory_chunk_tokens(0, False, seqs, n * seqs, n, 8, 128, 256, True, **kw)  # noqa: E731
    assert tokens(47) == 0 and tokens(48) == 32 and tokens(128) == 32 and tokens(129) == 64
    assert tokens(23, 4) == 0 and tokens(24, 4) == 32 and tokens(33, 4) == 64 and tokens(47, 3) == 0
    # chunk states stay within their limit: longer chunks then, which are walked
    many = tokens(2000, 64)
    assert many > 64 and 64 * -(-2000 // many) * 8 * 128 * 256 * 4 <= 2 * ops.MEMORY_CHUNKS_MAX_BYTES
    # without products as before
    assert ops.memory_chunk_tokens(0, False, 1, 100, 100, 8, 128, 256) == 0 and ops.memory_chunk_tokens(3, False, 1, 100, 100, 8, 128, 64) == 0


def test_single_tokens_beside_a_run():
    """Runs of one token pay for a whole chunk: a prompt beside many of them is walked token by token, one beside few is not."""
    from gopherllm_b200 import ops
    gated = lambda n, lone: ops.memory_chunk_tokens(0, False, 1 + lone, n + lone, n, 8, 128, 256, True)  # noqa: E731
    decay = lambda n, lone: ops.memory_chunk_tokens(3, False, 1 + lone, n + lone, n, 64, 128, 64, True)  # noqa: E731
    assert gated(24, 63) == gated(48, 15) == gated(128, 63) == gated(256, 63) == 0 and gated(128, 15) == gated(1000, 63) == 64
    assert decay(24, 15) == decay(128, 63) == decay(256, 63) == decay(500, 63) == 0 and decay(256, 15) == decay(300, 0) == 64
    assert ops.memory_chunk_tokens(0, False, 16, 4800, 300, 8, 128, 256, True) == 64
