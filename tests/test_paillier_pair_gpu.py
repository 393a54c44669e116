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
    """Counts of one item, a partial CTA, the last batch of the small rule
    (items per CTA at five limbs a lane, one CTA on every SM) and the first
    beyond it, for factors of `bits` bits at the top of their width."""
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
    for count in (1, items + 1, edge, edge + 1):
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
