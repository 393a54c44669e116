"""The benchmark's count of a search's transforms (no GPU): against a walk
through the circuit, tile by tile and merge by merge."""

import pytest


@pytest.mark.parametrize("tiles,padded,T,L,D,R", [(1024, 512, 7, 3, 6, 9), (11, 8, 7, 3, 6, 3), (1, 4, 3, 2, 4, 2),
                                                  (5, 2, 5, 2, 15, 1)])
def test_residue_transforms_count_the_circuit(tiles, padded, T, L, D, R):
    from bench import residue_transforms

    forward = inverse = 0
    read_by_composition = set()  # switches whose component 1 a later one composes from coefficients
    nodes = []
    for tile in range(tiles):
        forward += 2 * T + 3 * L
        inverse += 3 * T
        switches = [("tile", tile, k) for k in range(1 + R)]
        forward += len(switches) * (D - 1) * L
        read_by_composition.update(switches[:-1])
        nodes.append(switches[-1])
    for start in range(0, tiles, padded):
        stack = []
        for node in nodes[start:start + padded]:
            size = 1
            while stack and stack[-1][1] == size:
                read_by_composition.add(node)
                node, size = ("merge", start, stack.pop()[0], node), 2 * size
                forward += (D - 1) * L
            stack.append((node, size))
        node = stack.pop()[0]
        while stack:
            read_by_composition.add(node)
            node = ("merge", start, stack.pop()[0], node)
            forward += (D - 1) * L
        inverse += 2 * L
    inverse += len(read_by_composition) * L
    assert residue_transforms(tiles, padded, T, L, D, R) == (forward, inverse)
