"""Tile circuits that stay in the coefficient domain (tile_circuit): gadgets of
one digit, tiles without rotations, and rotation lists with the identity,
against the same circuit put together from the primitives.  Integer work:
equality is exact."""

import pytest

from test_bfv_rotations_gpu import T, _circuit, _group, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,q_bits,digit_bits,embed,tiles", [
    (64, 60, 60, 5, 11),      # one digit of a word; merges of few pairs
    (128, 120, 120, 7, 75),   # one digit of two words; the mask in the last switch
    (64, 120, 30, 1, 3),      # one vector slot a row: no rotation, the mask by itself
])
def test_search_equals_the_circuit_of_primitives(n, q_bits, digit_bits, embed, tiles):
    m, lay, q, layout, ring, relin, keys, poly = _setup(n, q_bits, digit_bits, embed, n + tiles)
    query, index = (poly(), poly()), [(poly(), poly()) for _ in range(tiles)]
    target = format(lay.coefficient_modulus(50), "x")
    server = m.create_server(relin, tuple(keys.items()), layout.padded, T, target)

    def packed(ct):
        return tuple(lay.pack_poly(c, q.bit_length()) for c in ct)

    got = m.packed_search(server, packed(query), tuple(packed(ct) for ct in index), tiles * layout.capacity - 1, False)
    tile, merge = _circuit(m, lay, q, layout, ring, relin, keys, n)
    cts = [tile(query, ct, layout.capacity - (k + 1 == tiles)) for k, ct in enumerate(index)]
    assert got == [packed(_group(cts[k:k + layout.padded], merge)) for k in range(0, tiles, layout.padded)]


@pytest.mark.parametrize("exponents", [(), (1,), (1, 3), (3, 1), (3, 1, 9)])
def test_tile_with_the_identity_among_its_rotations(exponents):
    n = 64
    m, lay, q, layout, ring, relin, keys, poly = _setup(n, 120, 30, 5, 9)
    key = next(iter(keys.values()))  # any key serves: the circuit does not depend on its value
    query, t, mask = (poly(), poly()), (poly(), poly()), poly()
    width = (q.bit_length() + 7) // 8

    def raw(p):
        return lay.fixed_poly(p, q)

    def ints(b):
        return [int.from_bytes(b[i * width:(i + 1) * width], "little") for i in range(n)]

    def add(x, y):
        return tuple([(a + b) % q for a, b in zip(u, v)] for u, v in zip(x, y))

    diff = tuple([(a - b) % q for a, b in zip(u, v)] for u, v in zip(query, t))
    c0, c1, c2 = (ints(b) for b in m.multiply(ring, tuple(raw(c) for c in diff), None, T))
    ct = add((c0, c1), tuple(ints(b) for b in m.apply_key(relin, raw(c2))))
    for g in exponents:
        ct = add(ct, ct if g == 1 else tuple(ints(b) for b in m.rotate_rows(key, tuple(raw(c) for c in ct), g)))
    got = m.hamming_tile(relin, tuple(map(raw, query)), tuple(map(raw, t)), tuple((g, key) for g in exponents),
                         raw(mask), T)
    assert got == tuple(m.ring_product(ring, raw(c), raw(mask)) for c in ct)
