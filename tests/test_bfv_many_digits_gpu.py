"""Gadgets of one-bit digits: waves of few (op, prime) pairs whose digits are
more than a launch has rows for (18 tiles x 8 primes x 480 digits), and the last
wave that fits, against the same circuit put together from the primitives."""

import pytest

from test_bfv_rotations_gpu import T, _circuit, _group, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [17, 18])
def test_search_with_480_digits_equals_the_circuit_of_primitives(tiles):
    n = 16
    m, lay, q, layout, ring, relin, keys, poly = _setup(n, 480, 1, 3, tiles)
    query, index = (poly(), poly()), [(poly(), poly()) for _ in range(tiles)]
    target = format(lay.coefficient_modulus(50), "x")
    server = m.create_server(relin, tuple(keys.items()), layout.padded, T, target)

    def packed(ct):
        return tuple(lay.pack_poly(c, q.bit_length()) for c in ct)

    got = m.packed_search(server, packed(query), tuple(packed(ct) for ct in index), tiles * layout.capacity, False)
    tile, merge = _circuit(m, lay, q, layout, ring, relin, keys, n)
    cts = [tile(query, ct, layout.capacity) for ct in index]
    assert got == [packed(_group(cts[k:k + layout.padded], merge)) for k in range(0, tiles, layout.padded)]
