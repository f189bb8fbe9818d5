"""The original-weights layer's tensor-core products (mx_gate_up_*, mx_down_*) against the CPU oracle, on the card's own
picks and quantized rows, and every product against 64 bits on the card's own quantized vectors: tiles that are full,
ragged and of one row, widths whose last stage of 256 inputs is half empty, both storage forms of the always-on expert and
none."""
import ctypes as C

import numpy as np
import pytest

from anemone_b200 import records as R
from anemone_b200 import synthetic
from oracle.binding import ptr, u8p
from tests import mx_exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,capacity,hidden,inner,experts,picks,shared", [
    (8, 8, 640, 384, 12, 4, "block128"),  # the decode form, half stages
    (1, 8, 512, 128, 9, 2, "e8m0"),
    (33, 64, 256, 256, 6, 3, None),  # the decode form with several jobs an expert
    (257, 512, 2048, 128, 3, 1, None),  # many rows, a single block of 128 inputs in down
    (130, 160, 1152, 256, 5, 2, "e8m0"),  # 1152 = four stages and a half; an always-on tile of two rows
    (203, 256, 1024, 384, 12, 3, "block128"),  # ragged tiles, one of two and more; 384 = a stage and a half
    (9, 16, 1024, 512, 40, 8, "block128"),  # a row or two an expert
    (700, 700, 128, 128, 6, 2, "block128"),  # small matrices that many pairs bring here: a stage of one block, all through
    (345, 512, 256, 128, 12, 4, "e8m0"),
    (513, 513, 512, 384, 5, 2, None),
])
def test_layer_matches_oracle(oracle, rows, capacity, hidden, inner, experts, picks, shared):
    from anemone_b200 import api
    from anemone_b200.moe import MoeConfig
    from anemone_b200.mx import MxLayer, MxLayout
    from oracle import moe_reference
    wide = capacity > 64 or (shared is not None and capacity > 8)
    config = MoeConfig(hidden=hidden, inner=inner, experts=experts, shared=0 if shared is None else 1, picks=picks,
                       row_capacity=capacity, activation_limit=7.0)
    H, I, block128 = hidden, inner, shared == "block128"
    rng = np.random.default_rng(rows)
    matrices = [(synthetic.mx_matrix(rng, I, H), synthetic.mx_matrix(rng, I, H), synthetic.mx_matrix(rng, H, I))
                for _ in range(experts)]
    draw = synthetic.e4m3_block128_matrix if block128 else synthetic.e4m3_matrix
    always = None if shared is None else (draw(rng, I, H), draw(rng, I, H), draw(rng, H, I))
    tokens = synthetic.tokens(rng, rows, H)
    scores = rng.normal(0, 1, size=(rows, experts)).astype(np.float32)
    scores[:, 1] += 1.5  # one expert with many rows
    L = MxLayout(config, 1, 0, block128=block128, wide=wide)
    card = api.Card(0, L.arena_bytes)
    try:
        layer = MxLayer(card, config, matrices, slices=(1, 1), shared_matrices=always, block128=block128, wide=wide)
        layer.connect_local([layer])
        assert len(layer.expert_launches) == 2  # the tensor-core launches are the ones that run
        for _ in range(2):  # both parity slots
            result = layer.step(tokens, scores)
            assert not card.waits_expired()
        received = card.download(0, L.arena_bytes)
    finally:
        card.close()
    chosen, weights = moe_reference.route(oracle, config, scores)
    picked = received[L.picks:L.picks + rows * picks * 4].view(np.uint32).reshape(rows, picks)
    assert np.array_equal(picked, chosen)
    # the jobs of the oracle: expert ascending, rows ascending, eight to a job
    table = received[L.expert_table:L.expert_table + experts * 24].view(np.uint64)
    jobs = (R.ExpertJob * L.job_capacity)()
    job = 0
    for expert in range(experts):
        held = [(row, slot) for row in range(rows) for slot in range(picks) if chosen[row, slot] == expert]
        for first in range(0, len(held), 8):
            record = jobs[job]
            record.gate_offset, record.up_offset, record.down_offset = (int(x) for x in table[3 * expert:3 * expert + 3])
            record.expert, record.row_count = expert, min(8, len(held) - first)
            for column, (row, slot) in enumerate(held[first:first + 8]):
                record.pair_index[column] = row * picks + slot
                record.route_weight[column] = float(weights[row, slot])
            job += 1
    expected = received.copy()
    expected[L.jobs:L.jobs + L.job_capacity * 96] = np.frombuffer(bytes(jobs), dtype=np.uint8)
    at = L.at
    oracle.orc_mx_experts(C.byref(R.ExpertGateUp(L.jobs, at["codes"], at["exponents"], at["operands"], at["hidden"], I, H,
                                                 L.pairs, picks, 7.0, 0)),
                          C.byref(R.ExpertDown(L.jobs, at["hidden_codes"], at["hidden_exponents"], at["hidden_operands"],
                                               at["pair_output"], H, I, L.pairs, 0)),
                          L.job_capacity, 1, 1, at["hidden_codes"], at["hidden_exponents"], at["hidden_operands"],
                          ptr(expected, u8p))

    def outputs(image, where, count):
        return synthetic.from_bfloat16(image[where:where + count * H * 2].view(np.uint16)).reshape(count, H)

    def close(got, want):
        assert np.isfinite(got).all() and np.abs(want).max() > 0
        assert np.abs(got - want).max() <= max(2e-2, 2.0 ** -6 * np.abs(want).max())
        a, b = got.reshape(-1).astype(np.float64), want.reshape(-1).astype(np.float64)
        assert a @ b / (np.linalg.norm(a) * np.linalg.norm(b)) >= 0.9999
        # Sums in another order round a gate or an up to its other bfloat16 neighbour for about one value in a thousand,
        # and one in sixteen of those moves a hidden value by a step of E4M3 (2^-3.5 of it): 2^-3.5 sqrt(1e-3 / 16) is
        # 7e-4 of the outputs' norm; four times that for the few hundred vectors of the smallest case
        assert np.linalg.norm(a - b) <= 2.8e-3 * np.linalg.norm(b)
    got = outputs(received, at["pair_output"], rows * picks)
    close(got, outputs(expected, at["pair_output"], rows * picks))
    summed = np.zeros((rows, H), dtype=np.float32)
    for slot in range(picks):
        summed = (summed + got.reshape(rows, picks, H)[:, slot, :]).astype(np.float32)
    if shared is not None:
        S = L.shared_at
        gate_up = R.TrunkLinearQuantized((C.c_uint64 * 2)(L.shared_matrices[0], L.shared_matrices[1]),
                                         (C.c_uint64 * 2)(S["gate_output"], S["up_output"]), at["codes"], at["exponents"],
                                         at["operands"], (C.c_uint32 * 2)(I, I), H, rows)
        down = R.TrunkLinearQuantized((C.c_uint64 * 2)(L.shared_matrices[2], 0), (C.c_uint64 * 2)(S["output"], 0),
                                      S["hidden_codes"], S["hidden_exponents"], S["hidden_operands"],
                                      (C.c_uint32 * 2)(H, 0), I, rows)
        (oracle.orc_shared_expert_block128 if block128 else oracle.orc_shared_expert)(
            C.byref(gate_up), C.byref(R.TrunkHidden(S["gate_output"], S["up_output"], S["hidden"], I, 7.0)),
            C.byref(R.ActivationQuantize(S["hidden"], S["hidden_codes"], S["hidden_exponents"], S["hidden_operands"], I, 0)),
            C.byref(down), 1, 1, ptr(expected, u8p))
        joined = outputs(received, S["output"], rows)
        close(joined, outputs(expected, S["output"], rows))
        summed = (summed + joined).astype(np.float32)
    # row sums, the join and the reduction: bit for bit given what the card wrote
    assert np.array_equal(result, synthetic.to_bfloat16(np.float32(0.0) + summed))
    check_products(received, L, rows, chosen, weights, matrices, always, block128)


def check_products(received, L, rows, chosen, weights, matrices, always, block128):
    """Every expert's hidden vectors from the card's quantized rows, and its outputs from the card's hidden vectors, in 64
    bits, with the bound of FP32 sums."""
    H, I, picks, experts = L.config.hidden, L.inner_local, L.config.picks, L.config.experts

    def span(offset, count, dtype=np.uint8):
        return received[offset:offset + count * np.dtype(dtype).itemsize].view(dtype)
    row_values = mx_exact.vectors(mx_exact.from_stream_order(span(L.stream_codes, rows * H).reshape(rows, H)),
                                  span(L.at["exponents"], rows * H // 32).reshape(rows, H // 32))
    if L.wide:  # tiles of 128 vectors in operand order: 16 bytes of an input group a vector; 512 bytes of scales a block
        tiles = L.tile_sizes["codes"] // (128 * H)
        codes = span(L.tile_at["hidden_codes"], tiles * 128 * I).reshape(tiles, I // 16, 128, 16)
        codes = codes.transpose(0, 2, 1, 3).reshape(tiles, 128, I)
        scales = span(L.tile_at["hidden_exponents"], tiles * 4 * I).reshape(tiles, I // 128, 32, 4, 4)  # row % 32, row / 32
        scales = scales.transpose(0, 3, 2, 1, 4).reshape(tiles, 128, I // 32)
    else:
        pair_codes = span(L.at["hidden_codes"], L.pairs * I).reshape(L.pairs, I)
        pair_exponents = span(L.at["hidden_exponents"], L.pairs * I // 32).reshape(L.pairs, I // 32)

    def check(at_rows, route, hidden, exponents, gate, up, down, outputs):
        hidden = mx_exact.from_stream_order(hidden)
        mx_exact.check_hidden(hidden, exponents, gate, up, row_values[at_rows], route, 7.0)
        mx_exact.check_outputs(outputs, down, mx_exact.vectors(hidden, exponents))
    pair_outputs = synthetic.from_bfloat16(span(L.at["pair_output"], L.pairs * H, np.uint16)).reshape(L.pairs, H)
    tile = 0
    for expert in range(experts):
        at_rows, slots = np.nonzero(chosen == expert)
        if at_rows.size == 0:
            continue
        pairs = at_rows * picks + slots
        if L.wide:
            count = -(-at_rows.size // 128)
            hidden = codes[tile:tile + count].reshape(-1, I)[:at_rows.size]
            exponents = scales[tile:tile + count].reshape(-1, I // 32)[:at_rows.size]
            tile += count
        else:
            hidden, exponents = pair_codes[pairs], pair_exponents[pairs]
        gate, up, down = (mx_exact.mx_weights(data, o, i) for data, (o, i) in zip(matrices[expert],
                                                                                  ((I, H), (I, H), (H, I))))
        check(at_rows, weights[at_rows, slots], hidden, exponents, gate, up, down, pair_outputs[pairs])
    if always is None:
        return
    if L.wide:
        first, held = tiles - (L.config.row_capacity + 31) // 32, 32 if block128 else 128
        hidden = np.concatenate([codes[first + base // held, :min(held, rows - base)] for base in range(0, rows, held)])
        exponents = np.concatenate([scales[first + base // held, :min(held, rows - base)] for base in range(0, rows, held)])
    else:
        hidden = span(L.shared_at["hidden_codes"], rows * I).reshape(rows, I)
        exponents = span(L.shared_at["hidden_exponents"], rows * I // 32).reshape(rows, I // 32)
    gate, up, down = (mx_exact.e4m3_weights(data, o, i, block128) for data, (o, i) in zip(always, ((I, H), (I, H), (H, I))))
    outputs = synthetic.from_bfloat16(span(L.shared_at["output"], rows * H, np.uint16)).reshape(rows, H)
    check(np.arange(rows), np.ones(rows), hidden, exponents, gate, up, down, outputs)
