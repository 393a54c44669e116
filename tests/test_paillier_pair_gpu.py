"""Exponentiation mod m^2 on pairs of residues mod m (k_pair_crt,
k_pair_modexp): batch sizes on both sides of the lanes-per-value rule, and the
halved exponent of a textbook key where its shortcut does not apply (factors
that are not prime, values that share a factor with n).  Integer work:
equality is exact."""

import math
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 148


def _odd(rng, bits):
    return rng.getrandbits(bits) | 1 | (1 << (bits - 1))


def _decrypt(c, e, mult, n):
    return (pow(c, e, n * n) - 1) // n * mult % n


@pytest.mark.parametrize("bits,items", [(512, 32), (1024, 16), (2048, 8)])
def test_batches_around_the_lanes_rule(bits, items):
    """Counts of one item, a partial CTA, the last batch with the components on
    different lanes (half the items per CTA, one CTA on every SM) and the first
    beyond it, the last batch of the small rule (items per CTA at five limbs a
    lane) and the first beyond it, for factors of `bits` bits at the top of their width."""
    import torch

    from cuhepy_b200.paillier.gpu import PaillierDevice

    rng = random.Random(bits)
    p, q = (1 << bits) - 2 * rng.randrange(1, 1 << 40) - 1, _odd(rng, bits)
    while math.gcd(p, q) != 1:
        q -= 2
    n = p * q
    ctx = PaillierDevice(n)
    e, mult = rng.getrandbits(70) | 1, rng.randrange(n)
    ctx.set_secret(e, mult)
    ctx.set_factors(p, q)
    base = [0, 1, n * n - 1, p, q * q, n + 1] + [rng.randrange(n * n) for _ in range(31)]
    want = torch.from_numpy(ctx.limbs([_decrypt(c, e, mult, n) for c in base]).view(np.int32)).cuda()
    powers = torch.from_numpy(ctx.limbs([pow(c, e, n * n) for c in base]).view(np.int32)).cuda()
    limbs = torch.from_numpy(ctx.limbs(base).view(np.int32)).cuda()
    edge = SMS * items
    for count in (1, items + 1, edge // 2, edge // 2 + 1, edge, edge + 1):
        rows = torch.arange(count, device="cuda") % len(base)
        c = limbs[rows].contiguous()
        out = torch.full_like(c, -1)
        torch.cuda.synchronize()
        ctx.decrypt_array(c, out, count)
        ctx.synchronize()
        assert torch.equal(out, want[rows]), count
        ctx.modexp_array(c, e, out, count)
        ctx.synchronize()
        assert torch.equal(out, powers[rows]), count


@pytest.mark.parametrize("bits", [500, 1000])
def test_halved_exponent_with_factors_that_are_not_prime(bits):
    from cuhepy_b200.paillier.gpu import PaillierDevice

    rng = random.Random(bits)
    p, q = 15 * _odd(rng, bits - 4), 7 * 11 * _odd(rng, bits - 8)
    while math.gcd(p, q) != 1:
        q += 2 * 7 * 11
    n = p * q
    ctx = PaillierDevice(n)
    ctx.set_factors(p, q)  # the secret after the factors
    for e in ((p - 1) * (q - 1), (p - 1) * 9, p - 1, (q - 1) * (1 << 60)):
        mult = rng.randrange(n)
        ctx.set_secret(e, mult)
        values = [0, 1, n + 1, 3 * p, q, n] + [rng.randrange(n * n) for _ in range(40)]
        assert ctx.decrypt(values) == [_decrypt(c, e, mult, n) for c in values], e.bit_length()
        units = [1 + n * rng.randrange(n) for _ in range(20)]  # 1 mod p and q: the shortcut holds
        assert ctx.decrypt(units) == [_decrypt(c, e, mult, n) for c in units]


@pytest.mark.parametrize("chunk_len,embed", [(1024, 700), (1024, 1), (96, 200), (33, 31)])
def test_lookup_digits_of_embeddings_and_words(chunk_len, embed):
    """Embedding digits (even chunk lengths: 8 and 16 bits of the embedding a
    row, part rows, chunks past the table's digits) and plain digits (odd chunk
    lengths, sparse words) against the integer kernel's 8-bit digits."""
    from cuhepy_b200.paillier.gpu import PaillierDevice

    rng = random.Random(chunk_len)
    n = _odd(rng, 1000)
    ctx = PaillierDevice(n)
    message_chunks = 125 if chunk_len == 1024 else 7
    ctx.build_tables(n + 1 + rng.randrange(n * n - n - 2), message_chunks, [rng.randrange(n * n) for _ in range(19)])
    gen = np.random.default_rng(chunk_len)
    chunk_num = -(-2 * embed // chunk_len)
    count = 70
    bits = gen.integers(0, 2, size=(count, embed), dtype=np.uint8)
    bits[0], bits[1], bits[2, : embed // 2] = 0, 1, 0
    noise = gen.integers(0, 19, size=(count * chunk_num, 14), dtype=np.uint8)
    words = [0, 1, 1 << (8 * message_chunks - 1), 255 << 8] + [rng.getrandbits(8 * message_chunks) % n for _ in range(40)]
    idx = gen.integers(0, 19, size=(len(words), 14), dtype=np.uint8)
    results = []
    for fp64, wide in ((0, 0), (1, 0), (1, 2)):
        ctx.set_fp64(fp64)
        ctx.set_wide_table(wide)
        results.append((ctx.lookup_encrypt_bits(bits, chunk_len, chunk_num, noise), ctx.lookup_encrypt_ints(words, idx)))
    assert results[0] == results[1]
    assert results[0] == results[2]


def test_lookup_encrypt_large_call_and_capture():
    """A call large enough for the table of noise products equals small calls;
    a call captured in a graph before any table was made for its pipe uses
    what is there."""
    import torch

    from cuhepy_b200.paillier.gpu import PaillierDevice

    rng = random.Random(5)
    n = _odd(rng, 1023)
    ctx = PaillierDevice(n)
    ctx.build_tables(n + 2, 16, [rng.randrange(n * n) for _ in range(256)])
    gen = np.random.default_rng(5)
    count, embed = 8192 + 3, 60
    bits = torch.from_numpy(gen.integers(0, 2, size=(count, embed), dtype=np.uint8)).cuda()
    noise = torch.from_numpy(gen.integers(0, 256, size=(count, 14), dtype=np.uint8)).cuda()
    large = torch.zeros((count, ctx.words), dtype=torch.int32, device="cuda")
    small = torch.zeros_like(large)
    part = torch.zeros_like(large)
    torch.cuda.synchronize()
    for lo in range(0, count, 4096):
        rows = min(4096, count - lo)
        ctx.lookup_encrypt_bits_array(bits[lo:lo + rows], rows, embed, 1024, 1, noise[lo:lo + rows], small[lo:lo + rows])
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="global"):
        ctx.lookup_encrypt_bits_array(bits, count, embed, 1024, 1, noise, part)
    graph.replay()
    torch.cuda.synchronize()
    ctx.set_stream(None)
    ctx.lookup_encrypt_bits_array(bits, count, embed, 1024, 1, noise, large)
    ctx.synchronize()
    assert torch.equal(large, small) and torch.equal(part, small)
