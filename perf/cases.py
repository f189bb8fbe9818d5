"""The calls a server of this library's expert layers makes, as timed cases.

A case is one layer call of one rank: routing, the experts' products, the row sums and the (here one-rank) ordered
reduction to bfloat16, through the classes a program uses (anemone_b200.moe, .prefill, .mx). A layer is loaded once and
serves many calls, as in a server: states of one configuration share it and differ in their tokens and router scores.

Fields of a case
  path      exl3_decode   MoeLayer.step: trellis-coded experts, host rows in, bfloat16 rows out
            exl3_prefill  PrefillLayer: the same layer for many rows
            mx_decode     MxLayer.step: MXFP4 routed experts and an E4M3 always-on expert
            mx_prefill    MxLayer(wide=True).step: the same for many rows
  rows      live rows of the call; capacity: the rows the layer was prepared for
  hidden, inner, experts, picks: the layer's shape (inner: the columns this rank holds); one always-on expert
  ranks     exl3_prefill: the experts are shared out over this many ranks and this is one of them
  block128  mx: the always-on expert has one FP32 scale per 128 x 128 weights (else one E8M0 code per 32 x 32)
  staged    exl3_prefill: the caller keeps its rows in page-locked memory and makes one call (else ordinary arrays)
"""
import math

import numpy as np
import torch

from anemone_b200 import api, synthetic
from anemone_b200.moe import MoeConfig, MoeLayer, MoeLayout
from anemone_b200.mx import MxLayer, MxLayout
from anemone_b200.prefill import PrefillLayer, PrefillLayout, Share

WEIGHT_SEED = 20261125
POOL = 4  # distinct experts drawn for a stored width; an expert's bytes stand in the arena on their own all the same
STAGED_STATES = 5  # states of one staged prefill layer that may be alive at once


def case(name, path, rows, capacity, hidden=4096, inner=2048, experts=256, picks=8, ranks=1, block128=False,
         staged=False):
    made = {"path": path, "rows": rows, "capacity": capacity, "hidden": hidden, "inner": inner, "experts": experts,
            "picks": picks, "ranks": ranks, "block128": block128, "staged": staged}
    if name:
        made["name"] = name
    return made


def listed():
    return [
        # one user's token: nine experts, the shortest call there is; launches and host work count
        case("exl3 decode 1", "exl3_decode", 1, 8),
        # the benchmark's decode step: eight tokens, about 58 experts
        case("exl3 decode 8", "exl3_decode", 8, 8),
        # a busy server's decode step: every fourth expert sees more than one row
        case("exl3 decode 32", "exl3_decode", 32, 32),
        # the decode step of one rank of eight: an eighth of every expert's columns
        case("exl3 decode 8 of tp8", "exl3_decode", 8, 8, inner=256),
        # a long prompt on one card
        case("exl3 prefill 4096", "exl3_prefill", 4096, 4096, staged=True),
        # the same prompt on one rank of eight: 32 routed experts and an eighth of the always-on expert
        case("exl3 prefill 4096 of ep8", "exl3_prefill", 4096, 4096, ranks=8, staged=True),
        # an ordinary prompt: a ragged number of rows, most experts with a few of them
        case("exl3 prefill 413", "exl3_prefill", 413, 512),
        # original weights: one user's token
        case("mx decode 1", "mx_decode", 1, 8, block128=True),
        # original weights: the benchmark's decode step
        case("mx decode 8", "mx_decode", 8, 8, block128=True),
        # original weights: a few rows on one rank of eight, the other storage of the always-on expert
        case("mx decode 5 of tp8", "mx_decode", 5, 8, inner=256),
        # original weights: the benchmark's prompt
        case("mx prefill 2048", "mx_prefill", 2048, 2048, block128=True),
        # original weights: a ragged prompt on one rank of eight
        case("mx prefill 333 of tp8", "mx_prefill", 333, 512, inner=256),
    ]


def draw(rng):
    path = rng.choice(["exl3_decode", "exl3_prefill", "mx_decode", "mx_prefill"])
    # MxLayer takes up to eight rows with an always-on expert in its decode form, more in its wide form
    low, high = {"exl3_decode": (1, 64), "exl3_prefill": (65, 4096), "mx_decode": (1, 8), "mx_prefill": (9, 2048)}[path]
    rows = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    hidden = rng.choice([1024, 1536, 2048, 2560, 3072, 4096])
    inner = 128 * int(round(math.exp(rng.uniform(math.log(2), math.log(16)))))
    experts = rng.choice([32, 48, 64, 128, 160, 256])
    capacity = max(8, 1 << (rows - 1).bit_length())
    staged = path == "exl3_prefill" and rng.random() < 0.5
    return case("", path, rows, rows if staged else capacity, hidden, inner, experts, rng.choice([4, 6, 8]),
                rng.choice([1, 2, 4]) if path == "exl3_prefill" else 1, path.startswith("mx") and rng.random() < 0.5,
                staged)


# ---- the layer a case runs on: loaded once, kept while calls on its configuration follow one another ----

class Loaded:
    key = layer = slots = None


def config_of(c):
    limit = 7.0 if c["path"].startswith("mx") else 10.0
    return MoeConfig(hidden=c["hidden"], inner=c["inner"], experts=c["experts"], shared=1, picks=c["picks"],
                     row_capacity=c["capacity"], activation_limit=limit)


def share_of(c, config):
    return Share.expert_parallel(config, c["ranks"], 0) if c["ranks"] > 1 else Share.whole(config)


def widths_of(config):
    rng = np.random.default_rng([WEIGHT_SEED, 3])
    return np.concatenate([synthetic.expert_widths(rng, config.experts), [3] * config.shared]).astype(np.uint32)


def held_experts(c, config):
    """(global expert, stored width, intermediate columns) of what this rank holds, by local number"""
    share, widths = share_of(c, config), widths_of(config)
    return [(e, int(widths[e]), share.inner if e < config.experts else share.shared_inner)
            for e in share.experts(config)]


def exl3_pool(hidden, held):
    """Stored matrices by local expert, POOL different ones a (width, columns)."""
    drawn = {}
    for place, (_, width, inner) in enumerate(held):
        key = (width, inner, place % POOL)
        if key not in drawn:
            rng = np.random.default_rng([WEIGHT_SEED, width, inner, place % POOL])
            drawn[key] = (synthetic.exl3_matrix(rng, hidden, inner, width), synthetic.exl3_matrix(rng, hidden, inner, width),
                          synthetic.exl3_matrix(rng, inner, hidden, width))
        yield drawn[key]


def mx_pool(hidden, inner, count):
    drawn = []
    for place in range(count):
        if place < POOL:
            rng = np.random.default_rng([WEIGHT_SEED, inner, place])
            drawn.append((synthetic.mx_matrix(rng, inner, hidden), synthetic.mx_matrix(rng, inner, hidden),
                          synthetic.mx_matrix(rng, hidden, inner)))
        yield drawn[place % POOL]


def load(c):
    config = config_of(c)
    H, I = config.hidden, config.inner
    if c["path"].startswith("exl3"):
        held = held_experts(c, config)
        widths = np.array([width for _, width, _ in held], dtype=np.uint32)
        if c["path"] == "exl3_decode":
            layout = MoeLayout(config, widths, 1, 0)
            card = api.Card(0, layout.arena_bytes)
            layer = MoeLayer(card, config, widths, exl3_pool(H, held))
        else:
            share = share_of(c, config)
            layout = PrefillLayout(config, widths, share)
            slot = api.align(layout.input_bytes, 4096) + api.align(16 + c["capacity"] * H * 2, 4096)
            card = api.Card(0, layout.arena_bytes, staging_bytes=max(64 << 20, STAGED_STATES * slot if c["staged"] else 0))
            layer = PrefillLayer(card, config, widths, exl3_pool(H, held), share)
    else:
        wide = c["path"] == "mx_prefill"
        layout = MxLayout(config, 1, 0, block128=c["block128"], wide=wide)
        rng = np.random.default_rng([WEIGHT_SEED, 9])
        store = synthetic.e4m3_block128_matrix if c["block128"] else synthetic.e4m3_matrix
        card = api.Card(0, layout.arena_bytes)
        layer = MxLayer(card, config, mx_pool(H, I, config.experts), slices=(2, 2),
                        shared_matrices=(store(rng, I, H), store(rng, I, H), store(rng, H, I)),
                        block128=c["block128"], wide=wide)
    layer.connect_local([layer])
    card.wait()
    return layer


def layer_of(c):
    key = tuple(sorted((name, value) for name, value in c.items() if name not in ("name", "rows")))
    if Loaded.key != key:
        if Loaded.layer is not None:
            Loaded.layer.card.close()
        Loaded.key = Loaded.layer = None
        Loaded.layer, Loaded.slots, Loaded.key = load(c), list(range(STAGED_STATES)), key
    return Loaded.layer, Loaded.slots


class Slot:
    """A state's part of a staged layer's page-locked block, given back with the state."""

    def __init__(self, free):
        self.free, self.index = free, free.pop()

    def __del__(self):
        self.free.append(self.index)


# ---- one call ----

def scores_of(c, seed):
    """Router scores: N(0, 1); a prompt's on top of a Zipf(1.1) popularity of the experts in a fixed shuffled order."""
    rng = np.random.default_rng([seed, 1])
    scores = rng.standard_normal((c["rows"], c["experts"]), dtype=np.float32)
    if c["path"].endswith("prefill"):
        popularity = 1.0 / np.arange(1, c["experts"] + 1, dtype=np.float64) ** 1.1
        order = np.random.default_rng([WEIGHT_SEED, 12]).permutation(c["experts"])
        scores += np.log(popularity / popularity.mean())[order].astype(np.float32)
    return scores


def prepare(c, seed):
    layer, free = layer_of(c)
    rng = np.random.default_rng([seed, 2])
    tokens = synthetic.to_bfloat16(rng.standard_normal((c["rows"], c["hidden"]), dtype=np.float32))
    state = {"layer": layer, "tokens": tokens, "scores": scores_of(c, seed), "rows": c["rows"],
             "prefill": c["path"] == "exl3_prefill", "slot": None}
    if c["staged"]:
        state["slot"] = slot = Slot(free)
        size = api.align(layer.layout.input_bytes, 4096)
        state["input_at"] = slot.index * (size + api.align(16 + c["capacity"] * c["hidden"] * 2, 4096))
        state["result_at"] = state["input_at"] + size
        layer.stage(state["input_at"], tokens, state["scores"])
    return state


def run(state):
    layer = state["layer"]
    if state["slot"] is not None:
        bits = layer.call(state["input_at"], state["result_at"])
    elif state["prefill"]:
        layer.load(state["tokens"], state["scores"])
        layer.run()
        bits = layer.result(state["rows"])
    else:
        bits = layer.step(state["tokens"], state["scores"])
    return torch.from_numpy(bits).view(torch.bfloat16)


def work(c):
    """Every chosen expert's matrices once, the rows and scores in, the result out; the products of every chosen pair."""
    config = config_of(c)
    H, rows, picks = config.hidden, c["rows"], config.picks
    chosen = np.argpartition(-scores_of(c, 0), picks - 1, axis=1)[:, :picks]
    counts = np.bincount(chosen.reshape(-1), minlength=config.experts)
    total = rows * (H * 2 + config.experts * 4 + H * 2)
    flops = 0
    if c["path"].startswith("exl3"):
        for expert, width, inner in held_experts(c, config):
            pairs = rows if expert >= config.experts else int(counts[expert])
            if pairs:
                total += 2 * synthetic.matrix_bytes(H, inner, width) + synthetic.matrix_bytes(inner, H, width)
                flops += 6 * H * inner * pairs
    else:
        weights = 3 * H * config.inner
        total += int((counts > 0).sum()) * (weights // 2 + weights // 32) + weights
        flops = 2 * weights * (rows * picks + rows)
    return {"bytes": total, "flops": flops}


def tolerance(c):
    # bfloat16 results of FP32 sums (mx: of E4M3-quantized hidden values): one bfloat16 step is 2^-8 of a value
    return {"rel": 1e-2}
