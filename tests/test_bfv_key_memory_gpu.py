"""Device memory of compiled keys: the form that NTT-domain rotations read is
made for the keys of a search or a tile circuit only, and where there is no
memory for it the coefficient domain gives the same responses."""

import numpy as np
import pytest

from bfv_helpers import random_fixed_poly, random_packed_poly

pytestmark = pytest.mark.gpu

T = 65537


def _ring(n, q_bits, seed):
    from cuhepy_b200.bfv import _bfv_rns as m
    from cuhepy_b200.bfv import layout as lay

    q = lay.rns_modulus(n, q_bits)
    rng = np.random.default_rng(seed)
    ring = m.create_ring(n, format(q, "x"), 30, True, True, 2)

    def poly():  # below q by its top byte
        width = (q_bits + 7) // 8
        raw = rng.integers(0, 256, size=(n, width), dtype=np.uint8)
        raw[:, -1] = rng.integers(0, q >> 8 * (width - 1), size=n)
        return raw.tobytes()

    def polys():
        return tuple((poly(), poly()) for _ in range(-(-q_bits // 30)))

    return m, lay, q, rng, ring, polys


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_keys_of_the_primitives_are_held_once():
    m, _, q, rng, ring, polys = _ring(8192, 180, 1)
    data = polys()
    keys = [m.compile_key(ring, data)]  # the ring's tables and workspace
    poly = random_fixed_poly(rng, 8192, q)
    m.apply_key(keys[0], poly)
    before = _free()
    for _ in range(16):
        keys.append(m.compile_key(ring, data))
        m.apply_key(keys[-1], poly)
    # device memory is given out in units of 2 MB
    assert before - _free() <= 16 * (m.key_bytes(keys[0]) + (2 << 20))


def test_search_without_memory_for_the_second_form():
    import torch

    n, embed, tiles = 16384, 256, 3
    m, lay, q, rng, ring, polys = _ring(n, 300, 2)
    layout = lay.Layout(n, embed)
    data = {g: polys() for g in [0] + sorted(set(layout.left()) | set(layout.right()))}
    target = format(lay.coefficient_modulus(50), "x")

    def packed():
        return random_packed_poly(rng, n, q), random_packed_poly(rng, n, q)

    query, index = packed(), tuple(packed() for _ in range(tiles))
    count = tiles * layout.capacity - 1

    def server(reserve=None):
        compiled = {g: m.compile_key(ring, d) for g, d in data.items()}
        held = None
        if reserve is not None:
            held = torch.empty(_free() - reserve, dtype=torch.uint8, device="cuda")
        relin = compiled.pop(0)
        made = m.create_server(relin, tuple(compiled.items()), layout.padded, T, target)
        after = _free()
        del held
        torch.cuda.empty_cache()
        return made, relin, compiled, after

    lifted, *_ = server()
    want = m.packed_search(lifted, query, index, count, True)
    size = m.key_bytes(m.compile_key(ring, data[0]))
    reserve = size * 3 // 4
    plain, relin, keys, after = server(reserve)
    assert after > reserve // 2  # no key took its second form
    before = _free()
    assert m.packed_search(plain, query, index, count, True) == want
    # a tile circuit lifts the keys it uses, now that there is memory
    poly = tuple(random_fixed_poly(rng, n, q) for _ in range(5))
    rotations = tuple((g, keys[g]) for g in layout.left())
    first = m.hamming_tile(relin, poly[:2], poly[2:4], rotations, poly[4], T)
    assert m.hamming_tile(relin, poly[:2], poly[2:4], rotations, poly[4], T) == first
    assert before - _free() >= size * len(rotations)
