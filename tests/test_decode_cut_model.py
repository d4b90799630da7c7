"""CPU model of how the paged-decode kernel cuts its cost line into chunks (csrc/paged_decode.cu: Cut, make_cut): the
chunks tile the line, none is empty, the chunk of a unit is found again, every tile of every sequence is served once, and
the combine of a split sequence reads exactly the records written for it."""
import numpy as np
import pytest

TILE, ITEM_COST, MIN_CHUNK = 64, 3, 5


class Cut:
    def __init__(self, total, num_groups):
        self.groups = num_groups if total >= MIN_CHUNK * num_groups else max(total // MIN_CHUNK, 1)
        self.len, self.rem = divmod(total, self.groups)

    def bound(self, chunk):
        return chunk * self.len + min(chunk, self.rem)

    def chunk_of(self, u):
        head = self.rem * (self.len + 1)
        return u // (self.len + 1) if u < head else self.rem + (u - head) // self.len


@pytest.mark.parametrize("num_groups", [1, 2, 37, 74, 148, 296])
@pytest.mark.parametrize("ctx", [[1], [300], [64 * 5], [64 * 6, 0, 1], list(range(0, 4000, 37)), [32768] * 3 + [16] * 90,
                                 [131072], [700] * 120, [40] * 2000])
def test_chunks_tile_the_line_and_combines_read_what_was_written(ctx, num_groups):
    tiles = [-(-c // TILE) for c in ctx]
    units = [t + ITEM_COST if t else 0 for t in tiles]
    start = np.concatenate([[0], np.cumsum(units)]).tolist()
    cut = Cut(start[-1], num_groups)
    n = cut.groups
    bounds = [cut.bound(c) for c in range(n + 1)]
    assert bounds[0] == 0 and bounds[-1] == start[-1] and n <= num_groups
    assert all(a < b for a, b in zip(bounds, bounds[1:])), "an empty chunk would leave a ticket short"
    records, whole = {}, set()
    served = [np.zeros(t, int) for t in tiles]
    for c in range(n):
        assert cut.chunk_of(bounds[c]) == c and cut.chunk_of(bounds[c + 1] - 1) == c
        for b, t in enumerate(tiles):
            first = start[b] + ITEM_COST
            t0, t1 = (min(max(x - first, 0), t) for x in (bounds[c], bounds[c + 1]))
            if t0 < t1:
                served[b][t0:t1] += 1
                if t1 - t0 == t:
                    whole.add(b)
                else:
                    assert (c, int(t0 == 0)) not in records, "two results in one record"
                    records[(c, int(t0 == 0))] = b
    assert all((s == 1).all() for s in served)
    for b, t in enumerate(tiles):
        if t and b not in whole:
            first = start[b] + ITEM_COST
            gf, gl = cut.chunk_of(first), cut.chunk_of(first + t - 1)
            assert [k for k, v in records.items() if v == b] == [(c, int(c == gf)) for c in range(gf, gl + 1)]
        elif t:
            assert cut.chunk_of(start[b] + ITEM_COST) == cut.chunk_of(start[b] + ITEM_COST + t - 1)
