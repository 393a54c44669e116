"""Tile circuits and merges in the NTT domain (k_rotate_tm and its unfused
form) against the same circuit put together from the primitives, whose
switches run in the coefficient domain: sizes with and without a left-over
transform stage, few and many digits (summed unreduced up to seven), digits
wider than a word, and tile counts on both sides of the unfused rule (148
(op, prime) pairs).  Integer work: equality is exact."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

T = 65537


def _setup(n, q_bits, digit_bits, embed, seed):
    from cuhepy_b200.bfv import _bfv_rns as m
    from cuhepy_b200.bfv import layout as lay

    q = lay.rns_modulus(n, q_bits)
    rng = np.random.default_rng(seed)
    layout = lay.Layout(n, embed)
    ring = m.create_ring(n, format(q, "x"), digit_bits, True, True, 2)

    def poly():
        return [int.from_bytes(rng.bytes(q_bits // 8 + 9), "little") % q for _ in range(n)]

    def key():
        return m.compile_key(ring, tuple((lay.fixed_poly(poly(), q), lay.fixed_poly(poly(), q))
                                         for _ in range(-(-q_bits // digit_bits))))

    relin = key()
    keys = {g: key() for g in sorted(set(layout.left()) | set(layout.right()))}
    return m, lay, q, layout, ring, relin, keys, poly


def _circuit(m, lay, q, layout, ring, relin, keys, n):
    """tile and merge functions over pairs of coefficient lists."""
    width = (q.bit_length() + 7) // 8

    def raw(p):
        return lay.fixed_poly(p, q)

    def ints(b):
        return [int.from_bytes(b[i * width:(i + 1) * width], "little") for i in range(n)]

    def add(x, y):
        return tuple([(a + b) % q for a, b in zip(u, v)] for u, v in zip(x, y))

    def rotate(ct, g):
        return tuple(ints(b) for b in m.rotate_rows(keys[g], tuple(raw(c) for c in ct), g))

    def tile(query, t, count):
        diff = tuple([(a - b) % q for a, b in zip(u, v)] for u, v in zip(query, t))
        c0, c1, c2 = (ints(b) for b in m.multiply(ring, tuple(raw(c) for c in diff), None, T))
        ct = add((c0, c1), tuple(ints(b) for b in m.apply_key(relin, raw(c2))))
        for g in layout.left():
            ct = add(ct, rotate(ct, g))
        mask = [int(v) for v in m.batch_encode(ring, T, layout.mask_slots(count))[0]]
        return tuple(ints(m.ring_product(ring, raw(c), raw(mask))) for c in ct)

    def merge(left, right, level):
        return add(left, rotate(right, layout.right()[level]))

    return tile, merge


def _group(cts, merge):
    stack = []
    for ct in cts:
        size, level = 1, 0
        while stack and stack[-1][1] == size:
            ct = merge(stack.pop()[0], ct, level)
            size, level = 2 * size, level + 1
        stack.append((ct, size))
    ct = stack.pop()[0]
    while stack:
        left, size = stack.pop()
        ct = merge(left, ct, size.bit_length() - 1)
    return ct


@pytest.mark.parametrize("n,q_bits,digit_bits,embed,tiles", [
    (64, 120, 30, 5, 11),    # whole radix-8 passes; partial groups
    (128, 120, 30, 7, 75),   # a left-over stage; 150 pairs: fused, merges of few pairs unfused
    (128, 120, 30, 8, 74),   # 148 pairs: unfused
    (64, 180, 12, 4, 52),    # 15 digits, fused
    (32, 180, 97, 3, 50),    # two digits wider than a word
])
def test_search_equals_the_circuit_of_primitives(n, q_bits, digit_bits, embed, tiles):
    m, lay, q, layout, ring, relin, keys, poly = _setup(n, q_bits, digit_bits, embed, n + tiles)
    query = (poly(), poly())
    index = [(poly(), poly()) for _ in range(tiles)]
    count = tiles * layout.capacity - 1
    server = m.create_server(relin, tuple(keys.items()), layout.padded, T, format(lay.coefficient_modulus(50), "x"))

    def packed(ct):
        return tuple(lay.pack_poly(c, q.bit_length()) for c in ct)

    got = m.packed_search(server, packed(query), tuple(packed(ct) for ct in index), count, False)
    tile, merge = _circuit(m, lay, q, layout, ring, relin, keys, n)
    cts = [tile(query, ct, layout.capacity - (k + 1 == tiles)) for k, ct in enumerate(index)]
    want = [packed(_group(cts[k:k + layout.padded], merge)) for k in range(0, tiles, layout.padded)]
    assert got == want


@pytest.mark.parametrize("n,q_bits,digit_bits,embed", [(8192, 180, 30, 512), (16384, 120, 60, 16)])
def test_tile_equals_the_circuit_of_primitives(n, q_bits, digit_bits, embed):
    m, lay, q, layout, ring, relin, keys, poly = _setup(n, q_bits, digit_bits, embed, n)
    query, t = (poly(), poly()), (poly(), poly())
    tile, _ = _circuit(m, lay, q, layout, ring, relin, keys, n)
    mask = lay.fixed_poly([int(v) for v in m.batch_encode(ring, T, layout.mask_slots(layout.capacity))[0]], q)
    got = m.hamming_tile(relin, tuple(lay.fixed_poly(c, q) for c in query), tuple(lay.fixed_poly(c, q) for c in t),
                         tuple((g, keys[g]) for g in layout.left()), mask, T)
    assert got == tuple(lay.fixed_poly(c, q) for c in tile(query, t, layout.capacity))
