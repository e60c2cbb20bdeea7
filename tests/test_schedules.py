"""Host-side restatement of the two device-side work schedules of the decode operators, checked for
the properties the kernels rely on (no GPU needed).

* MLA (csrc/decode_mla.cu, plan_here and the plan kernels, next_piece, slot_of, list_cuts): the units of all sequences, a start-up share and then one
  per 32 tokens, form one list; worker w of W takes the w-th of W equal consecutive ranges.  A piece of a sequence that a range
  boundary cuts leaves its result in slot 2 w, or 2 w + 1 if the sequence begins inside the range; the plan lists the
  cut sequences, from which alone the reduce kernel finds the pieces.
* GQA (csrc/decode_gqa.cu, plan_here and gqa_plan_kernel): the tokens of all sequences form one list, cut into equal
  consecutive ranges (a multiple of the 16-token tile); the pieces of sequences the ranges hold are
  listed in token order, so the pieces of a range, and the pieces of a sequence, are consecutive.
"""
import random

import pytest


SEQ_COST = 14      # units charged at the start of a sequence (kSeqCost)
PREFILL_SEQ_COST = 4
MAX_WORKERS = 96   # entries of the table of cut sequences


def mla_segments(lens, workers, tile=32, seq_cost=SEQ_COST):
    """Pieces as every role of a worker walks them: (worker, sequence, first unit, units, whole, where the sequence begins)."""
    tiles = [(n + tile - 1) // tile for n in lens]
    prefix = [0]
    for t in tiles:
        prefix.append(prefix[-1] + (t + seq_cost if t else 0))
    total = prefix[-1]
    per = (total + workers - 1) // workers if total > 0 else 1
    segments = []
    for w in range(workers):
        at, stop = w * per, min(total, (w + 1) * per)
        if at >= stop:
            continue
        lo, hi = 0, len(lens)
        while hi - lo > 1:                   # largest b with prefix[b] <= at: where the cursor starts
            mid = (lo + hi) // 2
            if prefix[mid] <= at:
                lo = mid
            else:
                hi = mid
        b = lo
        while at < stop:
            while prefix[b + 1] <= at:       # sequences without units in between
                b += 1
            upto = min(prefix[b + 1], stop)
            first = max(at - prefix[b] - seq_cost, 0)
            n = upto - prefix[b] - seq_cost - first
            at = upto
            if n > 0:
                segments.append((w, b, first, n, first == 0 and upto == prefix[b + 1], prefix[b]))
    return segments, prefix, per, tiles


def slot_of(worker, seq_begin, per):
    return 2 * worker + (1 if seq_begin > worker * per else 0)


def mla_cuts(prefix, per, seq_cost):
    """The plan's list: (sequence, first and last worker, slot of the first piece)."""
    cuts = []
    for b in range(len(prefix) - 1):
        begin, end = prefix[b], prefix[b + 1]
        if begin < end:
            first, last = (begin + seq_cost) // per, (end - 1) // per
            if first < last:
                cuts.append((b, first, last, slot_of(first, begin, per)))
    return cuts


@pytest.mark.parametrize("seq_cost", [SEQ_COST, PREFILL_SEQ_COST])
@pytest.mark.parametrize("seed", range(12))
def test_mla_ranges_cover_every_tile_once_and_the_reduce_kernel_finds_the_pieces(seed, seq_cost):
    rng = random.Random(seed)
    batch = rng.choice([1, 2, 7, 32, 100, 400])
    lens = [rng.choice([0, 1, 31, 32, 33, 500, 4097, rng.randrange(0, 9000)]) for _ in range(batch)]
    workers = rng.choice([1, 2, 3, 37, 74, MAX_WORKERS])
    segments, prefix, per, tiles = mla_segments(lens, workers, seq_cost=seq_cost)
    covered = set()
    for w, b, first, n, _, _ in segments:
        assert n > 0 and first + n <= tiles[b]
        for t in range(first, first + n):
            assert (b, t) not in covered
            covered.add((b, t))
    assert len(covered) == sum(tiles)
    # writers: pieces of sequences that are not whole, each into a slot of its own
    written = {}
    for w, b, _, _, whole, seq_begin in segments:
        if not whole:
            slot = slot_of(w, seq_begin, per)
            assert slot not in written and 0 <= slot < 2 * workers
            written[slot] = b
    # reader: the slots that the list names are those, sequence by sequence
    cuts = mla_cuts(prefix, per, seq_cost)
    assert len(cuts) <= max(workers - 1, 0) and len(cuts) <= MAX_WORKERS
    read = {}
    for b, first, last, first_slot in cuts:
        for k in range(first, last + 1):
            slot = first_slot if k == first else 2 * k
            assert slot not in read
            read[slot] = b
    assert read == written
    assert {b for b, _, _, _ in cuts} == {b for _, b, _, _, whole, _ in segments if not whole}
    # equal shares: no worker has more than `per` units
    load = {}
    for w, _, _, n, _, _ in segments:
        load[w] = load.get(w, 0) + n
    assert max(load.values(), default=0) <= per


PIECE_COST = 32    # token units charged at the start of a sequence (kPieceCost)


def gqa_pieces(lens, ranges):
    total = sum(n + PIECE_COST for n in lens if n > 0)
    per = max(16, (((total + ranges - 1) // ranges) + 15) & ~15)
    items, range_first, range_count = [], [None] * ranges, [0] * ranges
    before = 0
    for b, n in enumerate(lens):
        if n == 0:
            continue
        start = before + PIECE_COST                      # where the sequence's tokens begin, in units
        first_range, count = start // per, (start + n - 1) // per - start // per + 1
        first = len(items)
        for k in range(count):
            range_start = (first_range + k) * per
            begin, end = max(start, range_start), min(start + n, range_start + per)
            r = first_range + k
            range_first[r] = len(items) if range_first[r] is None else min(range_first[r], len(items))
            range_count[r] += 1
            items.append((b, count, begin - start, first, end - start))
        before += n + PIECE_COST
    return items, range_first, range_count, per


@pytest.mark.parametrize("seed", range(5))
def test_gqa_ranges_partition_the_token_list(seed):
    rng = random.Random(100 + seed)
    lens = [rng.choice([0, 1, 15, 16, 17, 700, 4096, rng.randrange(0, 5000)]) for _ in range(rng.choice([1, 5, 64]))]
    ranges = rng.choice([1, 18, 148, 1184])
    items, range_first, range_count, per = gqa_pieces(lens, ranges)
    assert per % 16 == 0 and len(items) <= ranges + len(lens)
    # pieces of a sequence: consecutive entries, tiling it exactly
    for b, n in enumerate(lens):
        mine = [(i, it) for i, it in enumerate(items) if it[0] == b]
        assert [i for i, _ in mine] == list(range(mine[0][0], mine[0][0] + len(mine))) if mine else n == 0
        pos = 0
        for i, (_, count, begin, first, end) in mine:
            assert count == len(mine) and first == mine[0][0] and begin == pos and end > begin
            pos = end
        assert pos == n
    # pieces of a range: consecutive entries, every entry in exactly one range, no range above its share
    seen = []
    for r in range(ranges):
        if range_count[r]:
            seen.extend(range(range_first[r], range_first[r] + range_count[r]))
            units = sum(end - begin for _, _, begin, _, end in items[range_first[r]:range_first[r] + range_count[r]])
            assert units <= per
    assert seen == list(range(len(items)))
