"""CPU model of the tile bookkeeping of the prefill kernel (csrc/varlen_prefill.cu): which tokens of which heads the two Q tiles
of a work item hold (make_pack, make_item: (token, head) rows of one kv head), which 128-key tiles they visit, how many keys of
the last one the products go through and what the element mask leaves of them, whole or cut into runs, must cover exactly the
causal region -- key c is used for query position p iff c <= p -- of every head once; and the item lists (the plan kernel's, and
the one a short launch's CTAs find themselves) must contain every (sequence, token block) once, longest causal span first."""
import numpy as np
import pytest

TILE, SPLIT_TILES = 128, 8
WHOLE_KEYS = 11 * TILE  # sequences without a cached prefix are cut if they have more keys


def make_pack(group, lone=False):
    """`lone`: items of tile A alone (no sequence has tokens as far behind a block's first as dq)."""
    w = max(x for x in range(1, 9) if group % x == 0)
    heads = w if w % 2 else w // 2
    tokens = TILE // heads
    if lone:
        return dict(w=heads, heads=heads, tokens=tokens, dq=1 << 28, dh=0, span=tokens, per_kv=group // heads)
    return dict(w=w, heads=heads, tokens=tokens, dq=tokens if w % 2 else 0, dh=0 if w % 2 else heads,
                span=2 * tokens if w % 2 else tokens, per_kv=group // w)


def visible_keys(pack, length, prefix, q0, x):
    return prefix + min(length, q0 + x * pack["dq"] + pack["tokens"])


def make_item(pack, length, prefix, q0, r):
    """Item r of the token block at q0, for one kv head: [(first head, first token, K/V tiles)] of Q tiles A and B."""
    n_a = (visible_keys(pack, length, prefix, q0, 0) - 1) // TILE + 1
    n_b = (visible_keys(pack, length, prefix, q0, 1) - 1) // TILE + 1 if length - q0 > pack["dq"] else 0
    head = r * pack["w"]
    return [(head, q0, n_a), (head + pack["dh"], q0 + pack["dq"], n_b)]


def runs(pack, tiles, splits, prefix, len_k):
    """Runs of an item (load_item of SplitParams): per run its first K/V tile and the tiles Q tiles A and B visit there."""
    n_a, n_b = tiles
    n_kv, count = max(n_a, n_b), 1
    if n_a >= SPLIT_TILES and (prefix > 0 or len_k > WHOLE_KEYS):
        count = min(splits, n_a // (3 if pack["span"] > TILE else 2))
    out = []
    for c in range(count):
        j0, j1 = n_a * c // count, n_kv if c + 1 == count else n_a * (c + 1) // count
        out.append((j0, min(n_a, j1) - j0, min(n_b, j1) - j0 if n_b else 0))
    return out


def seen_keys(pack, length, prefix, q0, x, row, j0, n):
    """Keys that row `row` of Q tile x uses in the n tiles from tile j0 on: unmasked tiles whole, of the others the keys up to the
    row's limit, by chunks of 32 that the warp's rows need (counted from the run's first tile, as the kernel does).  All of them
    must be keys that the products have gone through."""
    prefix -= j0 * TILE
    first = q0 + x * pack["dq"]
    live = min(pack["tokens"], length - first)
    tok = lambda r: min(r // pack["heads"], live - 1)
    warp = row // 32 * 32
    keys = []
    for j in range(n):
        lim, lo, hi = (prefix + first - j * TILE + tok(r) for r in (row, warp, warp + 31))
        through = 16 * (-(-min(TILE, visible_keys(pack, length, prefix, q0, x) - (n - 1) * TILE) // 16)) if j == n - 1 else TILE
        if j < (prefix + first + 1) // TILE:
            seen = np.arange(TILE)  # a plain tile
        else:
            seen = [np.arange(32 * c, 32 * c + 32) for c in range(4) if 32 * c <= hi]
            seen = np.concatenate([c[c <= lim] if c[-1] > lo else c for c in seen] or [np.arange(0)])
        assert len(seen) == 0 or seen[-1] < through, "a score that was not computed"
        keys.append(j0 * TILE + j * TILE + seen)
    return np.concatenate(keys)


@pytest.mark.parametrize("lone", [False, True])
@pytest.mark.parametrize("group", [1, 2, 3, 4, 5, 6, 7, 8, 10, 11, 16])
@pytest.mark.parametrize("prefix", [0, 1, 127, 128, 1500, 2048])
@pytest.mark.parametrize("length", [1, 5, 127, 128, 129, 255, 256, 257, 300, 512, 513])
def test_tiles_and_masks_cover_exactly_the_causal_region(length, prefix, group, lone):
    pack = make_pack(group, lone)
    assert pack["heads"] * pack["tokens"] <= TILE
    for splits in (1, 3, 16):
        covered = {}
        for q0 in range(0, length, pack["span"]):
            item = make_item(pack, length, prefix, q0, 0)
            parts = runs(pack, (item[0][2], item[1][2]), splits, prefix, prefix + length)
            for x, (head, first, n_x) in enumerate(item):
                if n_x == 0:
                    assert first >= length
                    continue
                rows = min(pack["tokens"], length - first) * pack["heads"]
                for row in {r for r in (0, 1, 31, 32, 100, 127, rows - 1) if r < rows}:
                    p = first + row // pack["heads"]
                    keys = [seen_keys(pack, length, prefix, q0, x, row, j0, (n_a, n_b)[x]) for j0, n_a, n_b in parts]
                    assert all(len(k) for k in keys), "a run none of whose keys a row sees has no maximum"
                    assert np.array_equal(np.concatenate(keys), np.arange(prefix + p + 1)), (length, prefix, q0, x, row)
                for r in range(pack["per_kv"]):
                    h0 = make_item(pack, length, prefix, q0, r)[x][0]
                    for t in range(first, min(first + pack["tokens"], length)):
                        for h in range(h0, h0 + pack["heads"]):
                            covered[h, t] = covered.get((h, t), 0) + 1
        assert covered == {(h, t): 1 for h in range(group) for t in range(length)}, "every row of every head once"


def blocks_of(lens, span=TILE):
    return [(b, level) for b, n in enumerate(lens) for level in range(-(-n // span))]


def test_plan_orders_items_longest_span_first():
    lens, prefixes = [700, 256, 1, 1300, 0, 257], [0, 3000, 128, 0, 500, 127]
    # the plan kernel: histogram per level, bases assigned from the highest level down, any order inside a level
    levels = {(b, l): (prefixes[b] + min(lens[b], (l + 1) * TILE) - 1) // TILE for b, l in blocks_of(lens)}
    for b, l in levels:  # as many K/V tiles in front of its last one as the item of the block has
        n_kv = max(n for _, _, n in make_item(make_pack(2), lens[b], prefixes[b], l * TILE, 0))
        assert levels[b, l] == n_kv - 1
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
