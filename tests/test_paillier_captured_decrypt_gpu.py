"""A decryption captured in a CUDA graph reads its key's schedules at every
replay: installing the factors once more leaves them where they are."""

import math
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("textbook", [True, False])
def test_replay_after_the_factors_are_installed_again(textbook):
    import torch

    from cuhepy_b200.paillier.gpu import PaillierDevice

    rng = random.Random(11)

    def odd(bits):
        return rng.getrandbits(bits) | 1 | (3 << (bits - 2))

    p, q = odd(512), odd(512)
    while math.gcd(p, q) != 1:
        q -= 2
    n = p * q
    ctx = PaillierDevice(n)
    e = (p - 1) * (q - 1) if textbook else rng.getrandbits(280) | 1
    mult = rng.randrange(n)
    ctx.set_factors(p, q)
    ctx.set_secret(e, mult)
    values = [1 + n * rng.randrange(n) for _ in range(9)] + [rng.randrange(n * n) for _ in range(40)]
    want = torch.from_numpy(ctx.limbs([(pow(c, e, n * n) - 1) // n * mult % n for c in values]).view(np.int32)).cuda()
    c = torch.from_numpy(ctx.limbs(values).view(np.int32)).cuda()
    out = torch.zeros_like(c)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        ctx.decrypt_array(c, out, len(values))
    others = []
    for again in range(3):
        if again:
            ctx.set_factors(p, q)
            # what was given back, if anything, is taken by another key
            others.append(PaillierDevice(odd(1024)))
            others[-1].set_secret(rng.getrandbits(1024), 1)
        out.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want), again
    ctx.set_stream(None)
