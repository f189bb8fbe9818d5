"""A bounded wait that ran out on the card reaches the caller: every call that runs a layer's graph and waits for it reads
the words of the graph's kernel files and refuses the outputs. The wait that runs out is a push reduction whose peer never
arrives (its deadline is a millisecond), in a kernel file that every layer's graph uses too."""
import ctypes as C

import numpy as np
import pytest

from anemone_b200 import prefill, synthetic
from anemone_b200 import records as R
from anemone_b200.moe import LINE, MoeConfig, MoeLayer, MoeLayout
from anemone_b200.mx import MxLayer, MxLayout
from anemone_b200.prefill import PrefillLayer, PrefillLayout

pytestmark = pytest.mark.gpu
H, I, EXPERTS = 512, 256, 8


@pytest.fixture(scope="module")
def api():
    from anemone_b200 import api as module
    assert module.card_count() >= 1, "no CUDA device: the CUDA path cannot run and there is no fallback"
    return module


def config_of(rows, shared=1):
    return MoeConfig(hidden=H, inner=I, experts=EXPERTS, shared=shared, picks=2, row_capacity=rows, activation_limit=7.0)


def exl3_matrices(rng, experts):
    return [(synthetic.exl3_matrix(rng, H, I, 3), synthetic.exl3_matrix(rng, H, I, 3), synthetic.exl3_matrix(rng, I, H, 3))
            for _ in range(experts)]


def mx_matrices(rng, hidden, inner):
    return [(synthetic.mx_matrix(rng, inner, hidden), synthetic.mx_matrix(rng, inner, hidden),
             synthetic.mx_matrix(rng, hidden, inner)) for _ in range(EXPERTS)]


def moe(api, rng, rows, form="fused", one_graph=True):
    config, widths = config_of(rows), np.full(EXPERTS + 1, 3, dtype=np.uint32)
    layout = MoeLayout(config, widths, 1, 0, reduce_form=form)
    card = api.Card(0, layout.arena_bytes + (1 << 20))
    layer = MoeLayer(card, config, widths, exl3_matrices(rng, EXPERTS + 1), reduce_form=form)
    layer.step_graph = None if one_graph else -1  # the copies as kernels of the step's graph, or beside it
    return layer, layout, layer.step


def mx(api, rng, rows, wide, shared=0, hidden=H, inner=I):
    config = MoeConfig(hidden=hidden, inner=inner, experts=EXPERTS, shared=shared, picks=2, row_capacity=rows,
                       activation_limit=7.0)
    layout = MxLayout(config, 1, 0, block128=False, wide=wide)
    card = api.Card(0, layout.arena_bytes + (1 << 20))
    always = tuple(synthetic.e4m3_matrix(rng, o, i) for o, i in ((inner, hidden), (inner, hidden), (hidden, inner)))
    layer = MxLayer(card, config, mx_matrices(rng, hidden, inner), slices=(1, 1), wide=wide,
                    shared_matrices=always if shared else None)
    return layer, layout, layer.step


def prompt(api, rng, rows, monkeypatch, pieces):
    monkeypatch.setattr(prefill, "call_pieces", lambda *_: pieces)
    config, widths = config_of(rows), np.full(EXPERTS + 1, 3, dtype=np.uint32)
    layout = PrefillLayout(config, widths)
    card = api.Card(0, layout.arena_bytes + (1 << 20))
    layer = PrefillLayer(card, config, widths, exl3_matrices(rng, EXPERTS + 1))

    def call(tokens, scores):
        layer.stage(0, tokens, scores)
        return layer.call(0, api.align(layout.input_bytes, 4096)).copy()
    return layer, layout, call


FORMS = {
    "exl3 step": lambda api, rng, patch: (8, moe(api, rng, 8)),
    "exl3 step, copies beside the graph": lambda api, rng, patch: (8, moe(api, rng, 8, "pull", False)),
    "mx step": lambda api, rng, patch: (8, mx(api, rng, 8, False, shared=1)),
    "mx prompt": lambda api, rng, patch: (40, mx(api, rng, 64, True, shared=1, hidden=1024)),
    "mx prompt with a side run": lambda api, rng, patch: (40, mx(api, rng, 64, True, shared=1)),
    "exl3 prompt": lambda api, rng, patch: (256, prompt(api, rng, 256, patch, 1)),
    "exl3 prompt in pieces": lambda api, rng, patch: (512, prompt(api, rng, 512, patch, 2)),
}


def wait_runs_out(api, card, space):
    """One push reduction of two ranks on the card's own memory, the second of which never arrives."""
    width = 256
    peer_table, step, pairs, output, region = (api.align(space + at, 256) for at in (0, 512, 1024, 4096, 8192))
    stride, inbox = 16384, 2 * 2 * LINE
    card.fill(space, 0, 1 << 19)
    peers = (R.OrderedPeer * 2)()
    for rank in range(2):
        peers[rank].region_offset = region + rank * 2 * stride
    card.upload(peer_table, np.frombuffer(bytes(peers), dtype=np.uint8))
    for rank in range(2):
        card.peer_connect(card, 0, peer_table + 32 * rank)
    card.upload(step, np.frombuffer(bytes(R.StepBlock(1, 1, 0)), dtype=np.uint8))
    push = R.OrderedRowsPushDescription()
    push.arguments.push = R.OrderedPush(peer_table, region, 0, output, inbox, step, stride, 2_000_000, width * 4, width, 2,
                                        0, R.ORDERED_PUSH_FP32, 0, 0)
    push.arguments.pair_output_offset, push.arguments.width, push.arguments.pairs_per_row = pairs, width, 1
    push.arena_byte_count = card.arena_bytes
    lib, launch = api.library(), R.KernelLaunch()
    lib.ordered_rows_push_prepare.argtypes = [C.POINTER(R.OrderedRowsPushDescription), C.POINTER(api.BackendOperations),
                                              C.c_void_p, C.POINTER(R.KernelLaunch)]
    api.check(lib.ordered_rows_push_prepare(C.byref(push), card.ops_pointer, card.handle, C.byref(launch)), "push")
    card.run([launch])
    card.wait()
    assert card.expired_bits() == 1


@pytest.mark.parametrize("form", FORMS)
def test_a_wait_that_ran_out_refuses_the_result(api, monkeypatch, form):
    rng = np.random.default_rng(3)
    rows, (layer, layout, call) = FORMS[form](api, rng, monkeypatch)
    card = layer.card
    try:
        layer.connect_local([layer])
        tokens = synthetic.tokens(rng, rows, layer.config.hidden)
        scores = rng.normal(0, 1, size=(rows, EXPERTS)).astype(np.float32)
        first = call(tokens, scores)
        assert np.array_equal(call(tokens, scores), first) and first.any()
        # a graph of kernel files without such words goes on whatever the others met
        select, launch = R.StepInputSelect(layout.arena_bytes, 64, layout.arena_bytes + 64, layout.arena_bytes + 128, 1, 64), \
            R.KernelLaunch()
        api.check(api.library().step_input_select_prepare(C.byref(select), C.c_uint64(card.arena_bytes), card.ops_pointer,
                                                          card.handle, C.byref(launch)), "step_input_select_prepare")
        other = card.step_capture([launch], 0, 0, 0, layout.arena_bytes + 64, card.staging_bytes - 64, 64)
        wait_runs_out(api, card, api.align(layout.arena_bytes, 4096) + 4096)
        card.graph_run_wait(other)
        for _ in range(2):  # the words stay set while the card is open
            with pytest.raises(api.StatusError, match="wait ran out") as raised:
                call(tokens, scores)
            assert raised.value.status == R.STATUS_TIMED_OUT
        if hasattr(layer, "check_status"):  # what a caller of submit asks
            with pytest.raises(RuntimeError, match="wait ran out"):
                layer.check_status()
    finally:
        card.close()
