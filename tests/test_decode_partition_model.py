"""CPU model of the integer logic of the paged-decode kernel (csrc/paged_decode.cu): the stream-K cut of the tile
stream into per-CTA chunks (make_cut, modelled in test_decode_cut_model.py), the walk of a chunk (next_item), which chunks
emit a partial result into which workspace record, which chunks the producer says hold tiles of the sequence (TileMeta gf, gl),
how many tickets are drawn before it is combined, and which records the combining CTA reads back.  Property-tested against brute
force: every tile is served exactly once, every output row is written exactly once, the ticket count equals the
number of partials written, and the combine step reads exactly the slots that were written for its sequence."""
import numpy as np
from hypothesis import given, settings, strategies as st

from test_decode_cut_model import ITEM_COST, TILE, Cut


def tiles_of(ctx):
    return (ctx + TILE - 1) // TILE


def units_of(tb):
    return tb + ITEM_COST if tb > 0 else 0


def main_kernel_model(ctx, num_groups):
    """Returns (direct, partial, served, cut): direct = set of sequences written straight to `out`;
    partial[(chunk, slot)] = (b, t0, t1, gf, gl) with the chunks the producer writes beside the sequence's last tile."""
    tiles = [tiles_of(c) for c in ctx]
    units = [units_of(t) for t in tiles]
    start = [0] + np.cumsum(units).tolist()
    direct, partial = set(), {}
    served = [np.zeros(t, dtype=np.int32) for t in tiles]
    if start[-1] == 0:
        return direct, partial, served, None
    cut = Cut(start[-1], num_groups)
    for chunk in range(cut.groups):
        x0, x1 = cut.bound(chunk), cut.bound(chunk + 1)
        # the walk of the kernel: start at the sequence whose units contain x0, go on while sequences start before x1
        b = next(i for i in range(len(ctx)) if units[i] > 0 and start[i] <= x0 < start[i] + units[i])
        while b < len(ctx) and start[b] < x1:
            tb, first = tiles[b], start[b] + ITEM_COST
            t0, t1 = min(max(x0 - first, 0), tb), min(max(x1 - first, 0), tb)
            if t0 < t1:
                served[b][t0:t1] += 1
                if t1 - t0 == tb:
                    assert b not in direct
                    direct.add(b)
                else:
                    slot = 1 if t0 == 0 else 0
                    assert (chunk, slot) not in partial, "a CTA would overwrite one of its two partial records"
                    gf = chunk if t0 == 0 else cut.chunk_of(first)
                    gl = chunk if t1 == tb else cut.chunk_of(first + tb - 1)
                    partial[(chunk, slot)] = (b, t0, t1, gf, gl)
            b += 1
    return direct, partial, served, cut


def merge_model(gf, gl):
    """Records merge_sequence reads."""
    return [(g, 1 if g == gf else 0) for g in range(gf, gl + 1)]


@settings(max_examples=300, deadline=None)
@given(st.lists(st.integers(min_value=0, max_value=3000), min_size=1, max_size=40),
       st.sampled_from([1, 2, 3, 5, 18, 37, 74, 148, 296]))
def test_every_tile_once_and_merge_reads_what_was_written(ctx, num_groups):
    direct, partial, served, _ = main_kernel_model(ctx, num_groups)
    for b, sv in enumerate(served):
        assert np.all(sv == 1), "each tile of each sequence is streamed by exactly one CTA"
    by_seq = {}
    for record, (b, t0, t1, gf, gl) in partial.items():
        by_seq.setdefault(b, []).append((record, t0, t1, gf, gl))
    for b, c in enumerate(ctx):
        tb = tiles_of(c)
        if tb == 0:
            assert b not in direct and b not in by_seq  # zero-filled in the prologue
        elif b in direct:
            assert b not in by_seq, "a directly written row must not be merged again"
        else:
            pieces = sorted(by_seq[b])
            assert len({p[3:] for p in pieces}) == 1, "every CTA of a sequence names the same chunks"
            gf, gl = pieces[0][3:]
            assert merge_model(gf, gl) == [p[0] for p in pieces], (ctx, num_groups, b, pieces)
            assert len(pieces) == gl - gf + 1, "the ticket gl - gf is the last one drawn"
            # the pieces tile the sequence without gap or overlap
            spans = sorted(p[1:3] for p in pieces)
            assert spans[0][0] == 0 and spans[-1][1] == tb
            assert all(a[1] == n[0] for a, n in zip(spans, spans[1:]))


def test_cost_weights_even_out_ranges_with_many_short_sequences():
    """64 one-tile sequences followed by one of 640 tiles, two groups: by tiles alone the first group would take all the
    short sequences plus 288 tiles; with the boundary cost it takes them plus 191 tiles only."""
    direct, partial, served, cut = main_kernel_model([10] * 64 + [640 * 64], 2)
    assert cut.bound(2) == 64 * 4 + 643
    assert partial[(0, 1)][:3] == (64, 0, 191) and partial[(1, 0)][:3] == (64, 191, 640)


def test_known_shapes():
    # one tile, 37 groups: one chunk, nothing to merge
    direct, partial, served, cut = main_kernel_model([1], 37)
    assert direct == {0} and not partial and cut.groups == 1
    # one long sequence over 37 groups: every chunk serves a piece
    direct, partial, _, cut = main_kernel_model([32768], 37)
    assert not direct and len(partial) == 37
    assert partial[(0, 1)][3:] == (0, 36)
    # less than five units per CTA: fewer, longer chunks
    assert main_kernel_model([300], 37)[3].groups == 1 and main_kernel_model([1500], 37)[3].groups == 5
