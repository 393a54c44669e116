"""Client encryption into separate buffers (cuhe_bfv_encrypt_parts) against
the contiguous call, and the device's reading of the public key: packed sizes
with and without a part word, one and several threads' worth of output, and a
key coefficient equal to q refused wherever it stands."""

import ctypes
import random

import numpy as np
import pytest

from bfv_helpers import fixed
from oracle import bfv as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bits,count", [(16, 60, 3), (16, 480, 1), (256, 180, 2), (8192, 180, 23)])
def test_parts_equal_the_contiguous_call_and_keys_are_checked(n, bits, count):
    from cuhepy_b200.bfv import _bfv_rns as m

    params = ob.Params(n, 97 if n == 16 else 65537, bits, 30, 21)
    q, t = params.q, params.t
    ring = m.create_ring(n, format(q, "x"), params.gadget_bits, True, True, 2)
    r = random.Random(n + bits)
    polys = [[r.randrange(q) for _ in range(n)] for _ in range(2)]
    polys[0][0] = polys[1][n - 1] = q - 1
    pk = tuple(fixed(p, q) for p in polys)
    slots = np.array([[r.randrange(t) for _ in range(n)] for _ in range(count)], dtype=np.uint32)
    u = np.array([[r.randrange(3) - 1 for _ in range(n)] for _ in range(count)], dtype=np.int8)
    e = np.array([[[r.randrange(-9, 10) for _ in range(n)] for _ in range(2)] for _ in range(count)], dtype=np.int8)
    size = (n * q.bit_length() + 7) // 8
    out = ctypes.create_string_buffer(2 * count * size)
    assert m.lib().cuhe_bfv_encrypt(ring.ptr, b"".join(pk), t, slots.ctypes.data, u.ctypes.data, e.ctypes.data, count,
                                    out) == 0
    got = m.encrypt_packed(ring, pk, t, slots, u, e)
    assert b"".join(c0 + c1 for c0, c1 in got) == out.raw
    for poly, at in ((0, 0), (1, n - 1)):
        bad = [list(p) for p in polys]
        bad[poly][at] = q
        with pytest.raises(ValueError, match="Noncanonical"):
            m.encrypt_packed(ring, tuple(fixed(p, q) for p in bad), t, slots, u, e)
