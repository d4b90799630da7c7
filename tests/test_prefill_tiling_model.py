"""CPU model of the tile bookkeeping of the prefill kernel (csrc/varlen_prefill.cu): which rows of which head the two Q tiles
of a work item hold (make_item: 128 rows of two heads, or 256 rows of the last head of an odd group), which 128-key tiles they
visit and what the element mask leaves of them, whole or cut into runs, must cover exactly the causal region -- key c is used
for query position p iff c <= p -- of every head once; and the item lists (the plan kernel's, and the one a short launch's CTAs
find themselves) must contain every (sequence, row block) once, longest causal span first."""
import numpy as np
import pytest

TILE, MIN_RUN, SPLIT_TILES = 128, 4, 12


def make_item(length, prefix, q0, group, r):
    """Item r of the row block at q0, for one kv head: [(head, first row, K/V tiles)] of Q tiles A and B, or None."""
    h2 = 2 * r
    two = h2 + 1 < group
    dq, dh = (0, 1) if two else (TILE, 0)
    nk_total = -(-(prefix + length) // TILE)
    n_a = min(nk_total, (prefix + q0 + TILE - 1) // TILE + 1)
    n_b = n_a if two else (min(nk_total, (prefix + q0 + 2 * TILE - 1) // TILE + 1) if length - q0 > TILE else 0)
    if not two and (q0 // TILE) & 1:
        return None
    return [(h2, q0, n_a), (h2 + dh, q0 + dq, n_b)]


def runs(tiles, splits):
    """Runs of an item (load_item of SplitParams): per run its first K/V tile and the tiles Q tiles A and B visit there."""
    n_a, n_b = tiles
    n_kv, count = max(n_a, n_b), 1 if n_a < SPLIT_TILES else min(splits, n_a // MIN_RUN)
    out = []
    for c in range(count):
        j0, j1 = n_a * c // count, n_kv if c + 1 == count else n_a * (c + 1) // count
        out.append((j0, min(n_a, j1) - j0, min(n_b, j1) - j0 if n_b else 0))
    return out


def seen_keys(prefix, first_row, row, j0, n):
    """Keys that row `row` of the Q tile at first_row uses in the n tiles from tile j0 on: unmasked tiles whole, of the others
    the keys up to the row's limit (relative to the run's first tile, as the kernel counts)."""
    first_lim = prefix - j0 * TILE + first_row
    n_plain = max(0, min(n, (first_lim + 1) // TILE))
    keys = [np.arange(n_plain * TILE)]
    for j in range(n_plain, n):
        lim = first_lim - j * TILE + row
        keys.append(j * TILE + np.arange(TILE)[np.arange(TILE) <= lim])
    return j0 * TILE + np.concatenate(keys)


@pytest.mark.parametrize("group", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("prefix", [0, 1, 127, 128, 1500, 2048])
@pytest.mark.parametrize("length", [1, 5, 127, 128, 129, 255, 256, 257, 300, 512, 513])
def test_tiles_and_masks_cover_exactly_the_causal_region(length, prefix, group):
    for splits in (1, 3, 16):
        covered = {}
        for q0 in range(0, length, TILE):
            for r in range((group + 1) // 2):
                item = make_item(length, prefix, q0, group, r)
                if item is None:
                    continue
                parts = runs((item[0][2], item[1][2]), splits)
                for x, (head, first_row, n_x) in enumerate(item):
                    if n_x == 0:
                        assert first_row >= length
                        continue
                    for row in {0, 1, 31, 32, 100, 127, min(TILE, length - first_row) - 1}:
                        p = first_row + row
                        if not 0 <= p < length or row < 0:
                            continue  # rows past the sequence are computed on whatever the tile holds and never stored
                        keys = [seen_keys(prefix, first_row, row, j0, (n_a, n_b)[x]) for j0, n_a, n_b in parts]
                        assert all(len(k) for k in keys), "a run none of whose keys a row sees has no maximum"
                        assert np.array_equal(np.concatenate(keys), np.arange(prefix + p + 1)), (length, prefix, q0, x, row)
                    for t in range(first_row, min(first_row + TILE, length)):
                        covered[head, t] = covered.get((head, t), 0) + 1
        assert covered == {(h, t): 1 for h in range(group) for t in range(length)}, "every row of every head once"


def blocks_of(lens):
    return [(b, level) for b, n in enumerate(lens) for level in range(-(-n // TILE))]


def test_plan_orders_items_longest_span_first():
    lens, prefixes = [700, 256, 1, 1300, 0, 257], [0, 3000, 128, 0, 500, 127]
    # the plan kernel: histogram per level, bases assigned from the highest level down, any order inside a level
    levels = {(b, l): prefixes[b] // TILE + l for b, l in blocks_of(lens)}
    top = max(levels.values()) + 1
    order = [k for level in range(top - 1, -1, -1) for k, v in levels.items() if v == level]
    assert sorted(order) == sorted(blocks_of(lens)) and len(order) == len(set(order)) == 6 + 2 + 1 + 11 + 0 + 3
    spans = [levels[k] for k in order]
    assert spans == sorted(spans, reverse=True)
    assert len(order) <= sum(lens) // TILE + len(lens) + 1, "fits the workspace capacity the host computes"


@pytest.mark.parametrize("lens", [[87], [0, 5, 0], [300, 5, 256, 257, 31], [128] * 32, [1] * 31 + [0], [0] * 31 + [600], []])
@pytest.mark.parametrize("ctas", [1, 3, 64])
def test_short_launches_find_every_row_block_once_and_the_long_ones_first(lens, ctas):
    """Lane b of a warp has sequence b; item `at` is found level by level from the highest, and in a level by lane."""
    blocks = [-(-n // TILE) for n in lens] + [0] * (32 - len(lens))
    items, found = sum(blocks), []

    def item(at):
        level = max(blocks) - 1
        while at >= sum(n > level for n in blocks):
            at -= sum(n > level for n in blocks)
            level -= 1
        mine = [n > level and sum(x > level for x in blocks[:b]) == at for b, n in enumerate(blocks)]
        return mine.index(True), level

    for cta in range(ctas):
        found += [(at, item(at)) for at in range(cta, items, ctas)]
    order = [k for _, k in sorted(found)]
    assert sorted(order) == sorted(blocks_of(lens)) and len(set(order)) == len(order)
    levels = [level for _, level in order]
    assert levels == sorted(levels, reverse=True)


@pytest.mark.parametrize("pairs,per_pair,groups", [(1, 8, 1), (7, 8, 2), (5, 24, 4), (13, 6, 2), (3, 8, 8)])
def test_head_groups_take_every_item_once_and_a_groups_heads_together(pairs, per_pair, groups):
    """load_item: item -> (pair, item of the pair)."""
    per, found = per_pair // groups, []
    for idx in range(pairs * per_pair):
        first = idx // (pairs * per) * per
        rest = idx - first * pairs
        found.append((rest // per, first + rest % per))
    assert sorted(found) == [(p, r) for p in range(pairs) for r in range(per_pair)]
    for g in range(groups):
        part = found[g * pairs * per:(g + 1) * pairs * per]
        assert {r // per for _, r in part} == {g} and [p for p, _ in part] == sorted(p for p, _ in part)
