"""Places of a piece's rows in the whole expert-parallel pass, against a pass written out row by row."""
import numpy as np
import pytest
import torch

from moonshine_b200 import ep


@pytest.mark.parametrize("world,pieces,experts", [(1, 2, 4), (2, 2, 8), (4, 3, 8)])
def test_places_of_a_piece(world, pieces, experts):
    rng = np.random.default_rng(world * 10 + pieces)
    # routes[source][piece]: expert of each route, in route order
    routes = [[rng.integers(0, experts, rng.integers(0, 30)) for _ in range(pieces)] for _ in range(world)]
    counts = [torch.tensor(np.stack([np.bincount(routes[s][p], minlength=experts) for s in range(world)]))
              for p in range(pieces)]
    per = experts // world
    for rank in range(world):
        first = rank * per
        seen, place = np.zeros(experts, int), {}               # (expert, source, piece) -> places
        for s in range(world):
            for p in range(pieces):
                for e in routes[s][p]:
                    place.setdefault((e, s, p), []).append(seen[e])
                    seen[e] += 1
        for p in range(pieces):
            group_rows, blocks = ep.part_of_pass(counts, p, first, per)
            assert group_rows.tolist() == seen[first:first + per].tolist()
            for e in range(per):
                for s in range(world):
                    got = place.get((first + e, s, p), [])
                    start = int(blocks[e * world + s])
                    assert got == list(range(start, start + len(got)))
