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


def _pair(seed, message_chunks, entries, pipe=1):
    """A context with its tables installed for `pipe`, and one with the same
    tables that keeps to the integer kernel's 8-bit digits."""
    from cuhepy_b200.paillier.gpu import PaillierDevice

    rng = random.Random(seed)
    n = _odd(rng, 1000)
    g, noise = rng.randrange(2, n * n), [rng.randrange(n * n) for _ in range(entries)]
    contexts = []
    for fp64 in (pipe, 0):
        ctx = PaillierDevice(n)
        ctx.set_fp64(fp64)
        ctx.set_wide_table(0)
        ctx.build_tables(g, message_chunks, noise)
        contexts.append(ctx)
    return contexts


class _Call:
    """`count` embeddings of `embed` bits with their noise, and a place for the result."""

    def __init__(self, ctx, seed, count, embed, entries, chunk_len=CHUNK_LEN):
        import torch

        gen = np.random.default_rng([seed, embed])
        self.count, self.embed, self.chunk_len = count, embed, chunk_len
        self.bits = torch.from_numpy(gen.integers(0, 2, size=(count, embed), dtype=np.uint8)).cuda()
        self.noise = torch.from_numpy(gen.integers(0, entries, size=(count, 14), dtype=np.uint8)).cuda()
        self.out = torch.zeros((count, ctx.words), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()

    def enqueue(self, ctx):
        ctx.lookup_encrypt_bits_array(self.bits, self.count, self.embed, self.chunk_len, 1, self.noise, self.out)

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


@pytest.mark.parametrize("message_chunks", [4, 5])
def test_entry_of_the_digit_zero_is_taken_as_one(message_chunks):
    """A table whose entries of the digit zero are not one: every kind of row
    leaves them out, as the integer kernel does, whatever the neighbours of a
    warp look up."""
    from cuhepy_b200.paillier.gpu import PaillierDevice

    rng = random.Random(message_chunks)
    n = _odd(rng, 1000)
    n2 = n * n
    table = [[rng.randrange(2, n2) for _ in range(256)] for _ in range(message_chunks)]
    noise = [rng.randrange(n2) for _ in range(5)]
    ctx = PaillierDevice(n)
    ctx.set_tables(table, noise)
    plain = [0, 1, 256, 255 << 8, 7 << 16, 9 << 24] + [rng.getrandbits(8 * message_chunks) for _ in range(30)]
    plain += [m & ~(255 << 8 * (k % message_chunks)) for k, m in enumerate(plain)]
    idx = np.array([[rng.randrange(5) for _ in range(14)] for _ in plain], dtype=np.uint8)
    want = []
    for m, row in zip(plain, idx):
        x = 1
        for i in range(message_chunks):
            d = m >> 8 * i & 255
            x = x * table[i][d] % n2 if d else x
        for k in row:
            x = x * noise[int(k)] % n2
        want.append(x)
    # embeddings: plaintext bit 2 i is embedding bit last - i; odd chunk lengths take plain digits
    embed = 4 * message_chunks
    bits = np.array([[rng.randrange(2) if k % 3 else 0 for _ in range(embed)] for k in range(40)], dtype=np.uint8)
    bits[5, : embed // 2] = 0
    bits[6, embed // 2:] = 0
    bnoise = np.zeros((40, 14), dtype=np.uint8)
    bwant = []
    for row in bits:
        m = sum(int(b) << 2 * (embed - 1 - i) for i, b in enumerate(row))
        x = pow(noise[0], 14, n2)
        for i in range(message_chunks):
            d = m >> 8 * i & 255
            x = x * table[i][d] % n2 if d else x
        bwant.append([x])
    for fp64 in (1, 0):
        ctx.set_fp64(fp64)
        for wide in (0, 2):
            ctx.set_wide_table(wide)
            assert ctx.lookup_encrypt_ints(plain, idx) == want, (fp64, wide)
            for chunk_len in (8 * message_chunks, 8 * message_chunks + 1):
                assert ctx.lookup_encrypt_bits(bits, chunk_len, 1, bnoise) == bwant, (fp64, wide, chunk_len)
    assert ctx.g_table() == table


@pytest.mark.parametrize("fp64", [1, 0])
def test_a_capture_without_tables_of_its_pipe_builds_nothing(fp64):
    """Tables installed for the integer pipe, the limb pairs and the wide table
    first wanted inside a capture: the 8-bit words serve."""
    import torch

    ctx, plain = _pair(2, 16, 16, pipe=0)
    call = _Call(ctx, 2, 50, 60, 16)
    want = call.result(plain)
    ctx.set_fp64(fp64)
    ctx.set_wide_table(2)
    graph = _capture(ctx, call)
    assert torch.equal(_replay(graph, call), want)
    assert not ctx.wide_table_ready()
    assert torch.equal(call.result(ctx), want)
    assert ctx.wide_table_ready()
    assert torch.equal(_replay(graph, call), want)


def _key_1024(message_chunks, entries):
    from cuhepy_b200.paillier.gpu import PaillierDevice

    rng = random.Random(7)
    n = _odd(rng, 2047)
    ctx = PaillierDevice(n)
    ctx.set_wide_table(0)
    ctx.build_tables(n + 2, message_chunks, [rng.randrange(n * n) for _ in range(entries)])
    return ctx


def _held(before):
    import torch

    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0]


def test_mode_0_holds_no_noise_products():
    """256^2 products of noise entries (42 MB) come with a large call, and go with mode 0."""
    import torch

    ctx = _key_1024(16, 256)
    call, small = _Call(ctx, 1, 8192, 60, 256), _Call(ctx, 2, 40, 60, 256)
    small.result(ctx)
    call.out.clone()
    before = torch.cuda.mem_get_info()[0]
    want = call.result(ctx)
    assert _held(before) < 1 << 24
    ctx.set_wide_table(1)
    assert torch.equal(call.result(ctx), want)
    assert _held(before) >= 256 * 256 * 640
    ctx.set_wide_table(0)
    assert _held(before) < 1 << 24
    assert torch.equal(call.result(ctx), want)


def test_wide_tables_share_one_bound():
    """Tables for embeddings (2.5 GiB), digits (5 GiB) and words (4 GiB): a
    context of the default mode holds at most 8 GiB of them."""
    import torch

    ctx = _key_1024(256, 16)
    count = 1 << 16
    call = _Call(ctx, 1, count, 1024, 16, 2048)
    words, out = torch.zeros_like(call.out), torch.zeros_like(call.out)
    torch.cuda.synchronize()
    want = call.result(ctx)
    call.out.clone()
    before = torch.cuda.mem_get_info()[0]
    ctx.set_wide_table(1)
    for fp64, least in ((1, 7 << 30), (0, 7 << 30), (1, 7 << 30)):
        ctx.set_fp64(fp64)
        assert torch.equal(call.result(ctx), want)
        ctx.lookup_encrypt_ints_array(words, count, call.noise, out)
        ctx.synchronize()
        assert least < _held(before) < (8 << 30) + (64 << 20), fp64
    ctx.set_wide_table(0)
    assert _held(before) < 1 << 24


@pytest.mark.parametrize("fp64", [1, 0])
def test_contexts_with_tables_of_other_sizes_on_two_threads(fp64):
    """Calls whose blocks ask for much and for little shared memory, each on
    its own context and thread: neither one's launch meets the other's limit."""
    import threading

    import torch

    jobs = []
    for seed, chunks, embed in ((4, 128, 500), (5, 2, 8)):
        ctx, plain = _pair(seed, chunks, 4)
        call = _Call(ctx, seed, 3, embed, 4)
        want = call.result(plain)
        ctx.set_fp64(fp64)
        jobs.append((ctx, call, want))
    errors = []

    def work(ctx, call):
        try:
            for _ in range(5000):
                if errors:
                    break
                call.enqueue(ctx)
            ctx.synchronize()
        except Exception as error:  # reported by the main thread
            errors.append(error)

    threads = [threading.Thread(target=work, args=job[:2]) for job in jobs]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert not errors
    for ctx, call, want in jobs:
        assert torch.equal(call.out, want)
