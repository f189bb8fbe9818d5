"""A staged prompt call in pieces on several ranks, without a card: the layers are prepared on a fake backend, every rank's
pieces are decoded from the launches they would queue, and the reductions they hold (of different row counts, through the
same two slots, call after call) are walked in every order the signal lines allow, on the ranks' own offsets, with the
copies out as late as they may be. The kernels' steps are restated here (kernel_ordered_b200.cu: ordered_row_sum_publish,
ordered_reduce_bf16 with owner runs)."""
import ctypes as C
import random

import numpy as np
import pytest

from anemone_b200 import prefill
from anemone_b200 import records as R
from anemone_b200.moe import LINE, MoeConfig
from anemone_b200.prefill import PrefillLayer, PrefillLayout, Share
from oracle.binding import pointer_array, ptr, u16p
from tests.test_host_preparers import FakeBackend

READY, REDUCED, DONE, PREVIOUS = 0, LINE, 2 * LINE, 72


class FakeCard:
    def __init__(self, arena_bytes):
        self.fake, self.arena_bytes = FakeBackend(), arena_bytes
        self.ops_pointer, self.handle = C.pointer(self.fake.table), self.fake.card
        self.arena, self.graphs = np.zeros(arena_bytes, dtype=np.uint8), []

    def upload(self, offset, array):
        data = np.ascontiguousarray(array).reshape(-1).view(np.uint8)
        self.arena[offset:offset + data.size] = data

    def fill(self, offset, value, byte_count):
        self.arena[offset:offset + byte_count] = value

    def graph(self, launches):
        self.graphs.append(list(launches))
        return len(self.graphs) - 1

    def view(self, offset, count, dtype):
        return self.arena[offset:offset + count * np.dtype(dtype).itemsize].view(dtype)


def layers_of(monkeypatch, ranks, rows, count, split, experts=8, inner=512):
    config = MoeConfig(hidden=128, inner=inner, experts=experts, shared=1, picks=2, row_capacity=rows)
    if count is not None:
        monkeypatch.setattr(prefill, "call_pieces", lambda *_: count)
    layers = []
    for rank in range(ranks):
        share = split(config, ranks, rank)
        widths = np.full(len(share.experts(config)), 3, dtype=np.uint32)
        card = FakeCard(PrefillLayout(config, widths, share).arena_bytes)
        layers.append(PrefillLayer(card, config, widths, (), share, rank, ranks))
    return config, layers


def reduction_of(layer, graph):
    publish, reduce = layer.card.graphs[graph][-2:]
    return (R.OrderedRowSumPublish.from_buffer_copy(bytes(publish.argument)[:C.sizeof(R.OrderedRowSumPublish)]),
            R.OrderedReduceBf16.from_buffer_copy(bytes(reduce.argument)[:C.sizeof(R.OrderedReduceBf16)]))


@pytest.mark.parametrize("split", [Share.expert_parallel, Share.tensor_parallel])
@pytest.mark.parametrize("ranks,experts,inner", [(2, 8, 512), (3, 8, 512), (5, 8, 640), (8, 9, 1152)])
def test_ranks_agree_on_what_they_share(monkeypatch, split, ranks, experts, inner):
    """Whatever the ranks' shares: a rank stores its run of the result at ITS offsets in every rank's memory."""
    config, layers = layers_of(monkeypatch, ranks, 1030, 4, split, experts, inner)
    first = layers[0]
    for layer in layers:
        for name in ("peer_table", "region", "parity_stride", "slot_input", "status", "result"):
            assert getattr(layer.layout, name) == getattr(first.layout, name), (layer.rank, name)
        assert [piece[:2] for piece in layer.pieces] == [piece[:2] for piece in first.pieces]
        for (_, rows, graph), (_, _, others) in zip(layer.pieces, first.pieces):
            publish, reduce = reduction_of(layer, graph)
            for mine, theirs in zip((publish, reduce), reduction_of(first, others)):
                assert mine.collective.rank == layer.rank
                for name in ("region_offset", "input_offset", "output_offset", "parity_stride", "element_count",
                             "rank_count"):
                    assert getattr(mine.collective, name) == getattr(theirs.collective, name), name
            assert publish.collective.element_count == rows * config.hidden and reduce.mode == R.ORDERED_REDUCE_OWNER_RUNS
    bounds = [piece[0] for piece in first.pieces] + [1030]
    assert bounds[0] == 0 and all(b % 128 == 0 for b in bounds[:-1])
    assert [piece[1] for piece in first.pieces] == list(np.diff(bounds))


@pytest.mark.parametrize("ranks", [2, 3, 8])
@pytest.mark.parametrize("rows,held", [(512, 256), (4096, 256), (4096, 32), (1030, 8)])
def test_ranks_agree_on_the_pieces(ranks, rows, held):
    """The estimate itself, from what every rank knows: the same count on every rank, by experts and by columns."""
    config = MoeConfig(hidden=4096, inner=2048, experts=held * ranks, shared=1, picks=8, row_capacity=rows)
    for split in (Share.expert_parallel, Share.tensor_parallel):
        counts = {prefill.call_pieces(config, split(config, ranks, rank), ranks) for rank in range(ranks)}
        assert len(counts) == 1 and counts <= {1, 2, 4}


@pytest.mark.parametrize("rows,experts,counts", [
    (512, 64, (1, 1, 1)), (1024, 64, (1, 1, 1)), (2048, 64, (1, 2, 2)), (4096, 64, (2, 2, 2)),
    (512, 256, (1, 1, 1)), (1024, 256, (1, 1, 1)), (2048, 256, (1, 1, 1)), (4096, 256, (1, 1, 2))])
def test_pieces_of_several_ranks(rows, experts, counts):
    """What is measured on one card decides nothing for 2, 4 and 8 ranks, whose pieces hold a reduction each."""
    config = MoeConfig(hidden=4096, inner=2048, experts=experts, shared=1, picks=8, row_capacity=rows)
    for split in (Share.expert_parallel, Share.tensor_parallel):
        assert tuple(prefill.call_pieces(config, split(config, ranks, 0), ranks) for ranks in (2, 4, 8)) == counts


@pytest.mark.parametrize("rows,experts,held,count", [(4096, 256, 32, 2), (4096, 256, 64, 2), (4096, 256, 128, 2),
                                                     (4096, 256, 256, 1), (1024, 256, 64, 1)])
def test_pieces_of_one_rank(rows, experts, held, count):
    """The fastest of 1, 2 and 4 pieces where they were timed."""
    config = MoeConfig(hidden=4096, inner=2048, experts=experts, shared=1, picks=8, row_capacity=rows)
    assert prefill.call_pieces(config, Share.expert_parallel(config, experts // held, 0), 1) == count


def walk(layers, calls, values, rng):
    """Runs the ranks' calls as coroutines, one random step at a time; returns [rank][call] the results. A coroutine yields
    False while it waits."""
    ranks = range(len(layers))
    arenas = [layer.card.view for layer in layers]
    results = [[None] * calls for _ in ranks]
    tasks = []

    def slot(record, at, rank, sequence):
        """Where `rank`'s slot lies, as the rank that holds `record` reaches it: its own peer table says so."""
        table = (R.OrderedPeer * len(layers)).from_buffer_copy(
            arenas[at](record.peer_table_offset, 32 * len(layers), np.uint8).tobytes())
        return table[rank].region_offset + (sequence & 1) * record.parity_stride

    def line(record, at, rank, sequence, phase):
        return arenas[rank](slot(record, at, rank, sequence) + phase, 1, np.uint64)

    def out_copy(me, layer, record, first, rows, into, finished):
        for _ in range(rng.randrange(40)):
            yield True
        H = layer.config.hidden
        assert arenas[me](record.status_offset, 1, np.uint32)[0] == 0
        into[first * H:(first + rows) * H] = arenas[me](record.collective.output_offset, rows * H, np.uint16)
        finished.append(first)

    def one_rank(me, layer):
        H, sequence = layer.config.hidden, 0
        for call in range(calls):
            into, finished = np.zeros(layer.config.row_capacity * H, dtype=np.uint16), []
            for first, rows, graph in layer.pieces:
                publish, reduce = reduction_of(layer, graph)
                c = publish.collective
                sequence += 1
                live = min(rows, c.element_count // H)
                arenas[me](publish.pair_output_offset, rows * H, np.float32)[:] = values[call][me][first * H:(first + rows) * H]
                yield True
                mine = slot(c, me, me, sequence)
                previous = int(arenas[me](mine + PREVIOUS, 1, np.uint64)[0])
                while previous != 0 and any(int(line(c, me, r, sequence, DONE)[0]) < previous for r in ranks):
                    yield False
                rows_out = arenas[me](mine + c.input_offset, live * H, np.float32)
                rows_in = arenas[me](publish.pair_output_offset, live * H, np.float32)
                for part in np.array_split(np.arange(live * H), 3):
                    rows_out[part] = np.float32(0.0) + rows_in[part]
                    yield True
                arenas[me](mine + PREVIOUS, 1, np.uint64)[0] = sequence
                line(c, me, me, sequence, READY)[0] = sequence
                yield True
                while any(int(line(c, me, r, sequence, READY)[0]) != sequence for r in ranks):
                    assert all(int(line(c, me, r, sequence, READY)[0]) <= sequence for r in ranks)
                    yield False
                vectors = live * H // 4
                share, longer = vectors // len(layers), vectors % len(layers)
                begin = me * share + min(me, longer)
                end = begin + share + (1 if me < longer else 0)
                for part in np.array_split(np.arange(4 * begin, 4 * end), 3):
                    total = np.zeros(part.size, dtype=np.float32)
                    for r in ranks:
                        total = total + arenas[r](slot(c, me, r, sequence) + c.input_offset, live * H, np.float32)[part]
                    bits = total.view(np.uint32).astype(np.uint64)
                    rounded = ((bits + 0x7FFF + ((bits >> 16) & 1)) >> 16).astype(np.uint16)
                    for r in ranks:
                        arenas[r](reduce.collective.output_offset, live * H, np.uint16)[part] = rounded
                    yield True
                line(c, me, me, sequence, REDUCED)[0] = sequence
                yield True
                while any(int(line(c, me, r, sequence, REDUCED)[0]) != sequence for r in ranks):
                    yield False
                line(c, me, me, sequence, DONE)[0] = sequence
                tasks.append(out_copy(me, layer, reduce, first, rows, into, finished))
                yield True
            while len(finished) < len(layer.pieces):  # the call returns when its last copy is made
                yield False
            results[me][call] = into
    tasks.extend(one_rank(me, layer) for me, layer in enumerate(layers))
    waited = 0
    while tasks:
        task = rng.choice(tasks)
        try:
            waited = 0 if next(task) else waited + 1
        except StopIteration:
            tasks.remove(task)
            waited = 0
        assert waited < 10000, "no rank can go on"
    return results


@pytest.mark.parametrize("ranks,rows,count", [(2, 519, 2), (2, 1100, 4), (3, 1030, 4), (5, 530, 2)])
def test_pieces_through_the_same_slots(oracle, monkeypatch, ranks, rows, count):
    calls = 3
    for seed in range(4):
        config, layers = layers_of(monkeypatch, ranks, rows, count, Share.expert_parallel)
        values = [[np.random.default_rng([seed, call, rank]).normal(0, 1, rows * config.hidden).astype(np.float32)
                   for rank in range(ranks)] for call in range(calls)]
        results = walk(layers, calls, values, random.Random(seed))
        for call in range(calls):
            want = np.zeros(rows * config.hidden, dtype=np.uint16)
            oracle.orc_ordered_reduce_bf16(pointer_array(values[call]), ranks, want.size, ptr(want, u16p))
            for rank in range(ranks):
                assert np.array_equal(results[rank][call], want), (seed, call, rank)
