"""The lookup encryption's tables over a context's life, against the integer
kernel's 8-bit digits on a context of its own.  Integer work: equality is
exact."""

import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNK_LEN = 1024


def _odd(rng, bits):
    return rng.getrandbits(bits) | 1 | (1 << (bits - 1))


def _pair(seed, message_chunks, entries):
    """A context and one with the same tables that keeps to the integer kernel's 8-bit digits."""
    from cuhepy_b200.paillier.gpu import PaillierDevice

    rng = random.Random(seed)
    n = _odd(rng, 1000)
    g, noise = rng.randrange(2, n * n), [rng.randrange(n * n) for _ in range(entries)]
    contexts = []
    for fp64 in (1, 0):
        ctx = PaillierDevice(n)
        ctx.set_fp64(fp64)
        ctx.set_wide_table(0)
        ctx.build_tables(g, message_chunks, noise)
        contexts.append(ctx)
    return contexts


class _Call:
    """`count` embeddings of `embed` bits with their noise, and a place for the result."""

    def __init__(self, ctx, seed, count, embed, entries):
        import torch

        gen = np.random.default_rng([seed, embed])
        self.count, self.embed = count, embed
        self.bits = torch.from_numpy(gen.integers(0, 2, size=(count, embed), dtype=np.uint8)).cuda()
        self.noise = torch.from_numpy(gen.integers(0, entries, size=(count, 14), dtype=np.uint8)).cuda()
        self.out = torch.zeros((count, ctx.words), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()

    def enqueue(self, ctx):
        ctx.lookup_encrypt_bits_array(self.bits, self.count, self.embed, CHUNK_LEN, 1, self.noise, self.out)

    def result(self, ctx):
        import torch

        self.out.zero_()
        torch.cuda.synchronize()
        self.enqueue(ctx)
        ctx.synchronize()
        return self.out.clone()


def _capture(ctx, call):
    import torch

    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="global"):
        call.enqueue(ctx)
    ctx.set_stream(None)
    return graph


def _replay(graph, call):
    import torch

    call.out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    return call.out.clone()


def test_wide_rows_grow_behind_a_captured_call():
    """Embeddings that reach 1, 3, 3, 8 and again 1 of the rows indexed by 16
    embedding bits: each call adds the rows it lacks, and a call captured with
    the first row alone replays to the same ciphertexts after every growth."""
    import torch

    ctx, plain = _pair(1, 32, 16)
    calls = [_Call(ctx, k, 45, embed, 16) for k, embed in enumerate((16, 48, 33, 128, 9))]
    want = [c.result(plain) for c in calls]
    ctx.set_wide_table(2)
    assert torch.equal(calls[0].result(ctx), want[0])
    assert ctx.wide_table_ready()
    graph = _capture(ctx, calls[0])
    for call, ciphertexts in zip(calls, want):
        assert torch.equal(call.result(ctx), ciphertexts), call.embed
        assert torch.equal(_replay(graph, calls[0]), want[0]), call.embed
    # a later capture reads all rows
    late = _capture(ctx, calls[3])
    assert torch.equal(_replay(late, calls[3]), want[3])
