"""Graphs with side runs and copy launches on a card (the reference's fork/join launch branches and BACKEND_COPY
nodes, source/backend_cuda_launch.c:486-632): the data that flows through copies on side runs into a kernel behind the
join, the same table run eagerly, and the refusals."""
import ctypes as C

import numpy as np
import pytest

from anemone_b200 import records as R

pytestmark = pytest.mark.gpu
WIDTH, SLOTS = 4096, 4


@pytest.fixture(scope="module")
def api():
    from anemone_b200 import api as module
    assert module.card_count() >= 1, "no CUDA device: the CUDA path cannot run and there is no fallback"
    return module


def row_sum_launch(api, card, pairs_offset, output_offset, arena_bytes, branch):
    record, launch = R.ExpertRowSum(pairs_offset, output_offset, WIDTH, SLOTS), R.KernelLaunch()
    api.check(api.library().bb_exl3_row_sum_prepare(C.byref(record), 1, arena_bytes, card.ops_pointer, card.handle,
                                                    C.byref(launch)), "bb_exl3_row_sum_prepare")
    launch.branch = branch
    return launch


def test_side_runs_and_copies(api):
    layout = api.Layout()
    row = WIDTH * 4
    sources = [layout.take(row) for _ in range(4)]
    pairs, other_pairs = layout.take(SLOTS * row), layout.take(SLOTS * row)
    output, other_output = layout.take(row), layout.take(row)
    arena_bytes = layout.take(0, 4096) + 4096
    card = api.Card(0, arena_bytes)
    try:
        rng = np.random.default_rng(12)
        values = [rng.normal(0, 1, WIDTH).astype(np.float32) for _ in range(4)]
        others = rng.normal(0, 1, (SLOTS, WIDTH)).astype(np.float32)
        table = [
            R.copy_launch(sources[0], pairs, row),                                  # 0 the main run
            R.copy_launch(sources[1], pairs + row, row, R.LAUNCH_SIDE),            # 1 a side run of two: behind 0
            R.copy_launch(pairs + row, pairs + 2 * row, row, R.LAUNCH_SIDE),       # 2 behind 1
            R.copy_launch(sources[3], pairs + 3 * row, row, R.LAUNCH_SIDE_MORE),   # 3 another side run: behind 0
            row_sum_launch(api, card, other_pairs, other_output, arena_bytes, R.LAUNCH_RESUME),  # 4 behind 0
            row_sum_launch(api, card, pairs, output, arena_bytes, R.LAUNCH_JOIN),  # 5 behind 2, 3 and 4
        ]
        want = np.zeros(WIDTH, dtype=np.float32)
        for term in (values[0], values[1], values[1], values[3]):
            want = want + term
        other_want = np.zeros(WIDTH, dtype=np.float32)
        for term in others:
            other_want = other_want + term
        graph = card.graph(table)
        for form in ("graph", "graph", "eager"):
            card.fill(0, 0, arena_bytes)
            for offset, value in zip(sources, values):
                card.upload(offset, value)
            card.upload(other_pairs, others)
            before = card.launch_count()
            if form == "graph":
                card.graph_run(graph)
            else:
                card.run(table)
            card.wait()
            assert card.launch_count() - before == 2  # the kernels; copies are no kernels
            assert np.array_equal(card.download(output, row, np.float32).view(np.uint32), want.view(np.uint32))
            assert np.array_equal(card.download(other_output, row, np.float32).view(np.uint32),
                                  other_want.view(np.uint32))
        # refusals: a table outside the grammar, a copy beyond the arena, a word nobody connected, an empty copy
        bad = list(table)
        bad[3] = R.copy_launch(sources[3], pairs + 3 * row, row, R.LAUNCH_RESUME)
        bad[4] = row_sum_launch(api, card, other_pairs, other_output, arena_bytes, R.LAUNCH_SIDE_MORE)
        graph_out = C.c_uint32(77)
        for broken in (bad, [R.copy_launch(sources[0], arena_bytes - 8, row)],
                       [R.copy_launch(sources[0], pairs, row, source_word=64)], [R.copy_launch(sources[0], pairs, 0)]):
            array = (R.KernelLaunch * len(broken))(*broken)
            assert card.ops.graph_capture(card.handle, array, len(array), C.byref(graph_out)) == R.STATUS_INVALID_ARGUMENT
            assert graph_out.value == 77
        for broken in ([R.copy_launch(sources[0], arena_bytes - 8, row)], [R.copy_launch(sources[0], pairs, 0)]):
            array = (R.KernelLaunch * len(broken))(*broken)
            assert card.ops.launch_run(card.handle, array, len(array)) == R.STATUS_INVALID_ARGUMENT
        # a copy through an address word: the card's own arena behind a word peer_connect wrote
        word = sources[2]
        card.peer_connect(card, pairs, word)
        card.upload(sources[0], values[2])
        card.run([R.copy_launch(sources[0], 2 * row, row, destination_word=word)])
        card.wait()
        assert np.array_equal(card.download(pairs + 2 * row, row, np.float32), values[2])
        beyond = (R.KernelLaunch * 1)(R.copy_launch(sources[0], arena_bytes - pairs - 8, row, destination_word=word))
        assert card.ops.launch_run(card.handle, beyond, 1) == R.STATUS_INVALID_ARGUMENT
    finally:
        card.close()


@pytest.mark.parametrize("sizes", [(1,), (63, 65, 17), ((1 << 19) - 1, (1 << 19) + 1), (1 << 20, 3, 5 << 20), (40 << 20,),
                                   (4 << 20,), ((4 << 20) - 5, 6), (8 << 20,), ((8 << 20) - 1, 2)])
def test_a_call_copies_ordinary_memory(api, sizes):
    """backend_b200_step_call without a graph: ranges of ordinary memory in and out again, at the edges of the pieces
    they are cut in (one piece, ragged ones, longer pieces where there would be too many), odd addresses and sizes."""
    rng = np.random.default_rng(len(sizes) + sizes[0])
    blocks = [rng.integers(0, 256, size=size + 3, dtype=np.uint8) for size in sizes]
    offsets = np.cumsum([0] + [api.align(size, 16) + 16 for size in sizes])
    card = api.Card(0, 64 << 20)
    try:
        for lead in (0, 3):
            card.fill(0, 0xA5, int(offsets[-1]))
            into = [block[lead:lead + size] for block, size in zip(blocks, sizes)]
            card.call(None, [(int(at), array) for at, array in zip(offsets, into)], [])
            back = [np.zeros(size + 3, dtype=np.uint8) for size in sizes]
            card.call(None, [], [(int(at), array[lead:lead + size]) for at, array, size in zip(offsets, back, sizes)])
            for array, sent, size, at in zip(back, into, sizes, offsets):
                assert np.array_equal(array[lead:lead + size], sent) and not array[:lead].any()
                assert (card.download(int(at) + size, 16) == 0xA5).all()  # nothing past the range
    finally:
        card.close()


def test_a_wait_is_for_its_own_run(api):
    """backend_b200_graph_run_wait behind runs of the same graph that graph_run left in the queue: it
    returns when ITS run's outputs are in place. Every run brings the pool's next entry, so the outputs say whose they
    are; the fills in front keep the earlier runs queued until the waiting one is."""
    entries, entry_bytes, earlier = 8, 4096, 5
    layout = api.Layout()
    pool, step, cursor = layout.take(entries * entry_bytes), layout.take(entry_bytes), layout.take(16)
    space_bytes = 1 << 30
    space = layout.take(space_bytes, 4096)
    card, lib = api.Card(0, layout.take(0, 4096) + 4096), api.library()
    try:
        for entry in range(entries):
            card.upload(pool + entry * entry_bytes, np.full(entry_bytes // 4, entry + 1, dtype=np.uint32))
        select, launch = R.StepInputSelect(pool, entry_bytes, step, cursor, entries, entry_bytes), R.KernelLaunch()
        lib.step_input_select_prepare.argtypes = [C.POINTER(R.StepInputSelect), C.c_uint64,
                                                  C.POINTER(api.BackendOperations), C.c_void_p,
                                                  C.POINTER(R.KernelLaunch)]
        api.check(lib.step_input_select_prepare(C.byref(select), card.arena_bytes, card.ops_pointer, card.handle,
                                                C.byref(launch)), "step_input_select_prepare")
        graphs = [card.step_capture([launch], 0, 0, 0, step, 4096 * which, entry_bytes) for which in (1, 3)]
        seen = [card.staging_view[4096 * which:4096 * which + entry_bytes].view(np.uint32) for which in (1, 3)]
        for turn in range(3):
            card.fill(cursor, 0, 16)
            for _ in range(20):  # several milliseconds
                card.fill(space, turn, space_bytes)
            for run in range(earlier):  # runs of both graphs among one another: a number is a graph's own
                card.graph_run(graphs[run % 2])
            card.graph_run_wait(graphs[0])
            assert (seen[0] == earlier + 1).all(), (turn, seen[0][0])
            card.graph_run_wait(graphs[1])
            assert (seen[1] == earlier + 2).all(), (turn, seen[1][0])
    finally:
        card.close()
