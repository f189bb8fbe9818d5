"""One rank's original-weights routed-expert layer (MXFP4 weights by E4M3 block-quantized activations), prepared once
and run per step through the C-ABI library. Launches of one step, all from libanemone_b200.so, where the widths are
multiples of 128 (tensor_products):
    mx_route_quantize -> mx_gate_up_few -> mx_down_few -> ordered_publish_reduce_flags_bf16
and for many rows
    exl3_prefill_picks -> exl3_prefill_group -> exl3_prefill_tiles -> mx_quantize -> mx_gather -> mx_gate_up_many
    -> mx_down_many -> expert_row_sum_entry -> trunk_rows_add_entry -> ordered_row_sum_publish -> ordered_reduce_bf16
(the last four as one launch, ordered_rows_one, where there is one rank)
(the products of the routed and the always-on experts on the fifth-generation tensor cores); otherwise
    router_select_b200 -> activation_quantize_entry -> expert_gate_up_<S> -> activation_quantize_entry (hidden)
    -> expert_down_<S> -> expert_row_sum_entry
    [-> trunk_linear_quantized_<S> (gate, up) -> trunk_hidden_entry -> activation_quantize_entry
     -> trunk_linear_quantized_<S> (down) -> trunk_rows_add_entry]          the always-on expert, E4M3 matrices
    -> ordered_row_sum_publish -> ordered_reduce_bf16
(linear_routed_experts_prepare's four, linear_shared_expert_prepare's four). Tensor parallelism is by intermediate columns, as in the
EXL3 decode layer; the ranks' FP32 rows are added in rank order and rounded once. Nothing here computes on the host.

wide=True is the same layer for MANY rows (the profile's prefill): the router's launch gives way to the three of
router_wide_prepare (the prefill's picks and grouping, then a job table of eight rows a job), the always-on expert to
linear_shared_expert_wide_prepare (a block column per eight rows), and the reduction adds by owner runs. The routed
experts' products are linear_routed_experts_wide_prepare's (a group of jobs and several tiles a block, the thin
instances' arithmetic; many=False keeps the thin instances, where every job streams its expert's matrices again).
"""
import ctypes as C

import numpy as np

from . import api
from . import records as R
from .moe import LINE, SIGNAL_BYTES, rank_columns

WEIGHT_FORMAT_E2M1_SCALED = 3
WEIGHT_FORMAT_E4M3_SCALED = 5
WEIGHT_FORMAT_E4M3_BLOCK128 = 6


# A prompt's products stay with mma.sync (group products) for matrices of fewer weights AND fewer (row, expert) pairs than
# these: the launches are then mostly their own beginnings and ends, and five smaller ones do it as fast as the three
# that set tensor memory up. The layer's graph, 12 to 256 experts of 2^14 to 2^17.6 weights: under 1024 pairs mma.sync
# takes 0.89 to 1.30 of the tensor cores' time (59 to 117 us), level in the middle, from 1024 pairs on 0.96 to 3.1 of it
# (256 experts, 512 x 256, top 8: 1024 rows 265 against 125 us). From 2^18 weights on 0.90 to 3.2 whatever the rows, 40 of
# 45 points above 1.05.
TENSOR_WIDE_WEIGHTS, TENSOR_WIDE_PAIRS = 1 << 18, 1024


def tensor_products(config, inner_local, wide, many):
    """Whether the products run on the fifth-generation tensor cores: whole blocks of 128 inputs and units of 128
    outputs, and for many rows matrices or rows that are worth it."""
    H = config.hidden
    worth_it = H * inner_local >= TENSOR_WIDE_WEIGHTS or config.row_capacity * config.picks >= TENSOR_WIDE_PAIRS
    return H % 128 == 0 and inner_local % 128 == 0 and (not wide or (many and worth_it))


def matrix_bytes(outputs, inputs):
    return outputs * inputs // 2 + outputs * inputs // 32


def shared_matrix_bytes(outputs, inputs, block128=False):
    """Stored bytes of an E4M3 matrix: one E8M0 code per 32 by 32 weights (the reference's format), or one FP32 scale
    per 128 by 128 (the original-weights checkpoints' block-scaled FP8)."""
    if block128:
        return outputs * inputs + (outputs + 127) // 128 * (inputs // 128) * 4
    return outputs * inputs + (outputs + 31) // 32 * (inputs // 32)


class MxLayout:
    def __init__(self, config, rank_count, rank, pool_entries=0, block128=False, wide=False):
        assert config.shared in (0, 1)
        self.block128, self.wide = block128, wide
        self.pool_entries = pool_entries
        self.config = c = config
        self.inner_local = I = rank_columns(c.inner, rank_count, rank)[1]
        H, rows = c.hidden, c.row_capacity
        self.pairs = pairs = rows * c.picks
        self.job_capacity = rows * c.picks // 8 + c.experts if wide else rows * c.picks
        layout = api.Layout()
        self.peer_table = layout.take(16 * 32)
        self.step = layout.take(256)
        self.tokens = layout.take(rows * H * 2)
        self.scores = layout.take(rows * c.experts * 4)
        self.step_input_bytes = layout.cursor - self.step
        # the status block stands directly in front of the result: one copy brings both back
        self.status = layout.take(16 + rows * H * 2)
        self.result = self.status + 16
        # optional: a pool of prepared step inputs resident on the card (step_input_select walks it)
        self.pool_stride = api.align(self.step_input_bytes, 256)
        self.cursor = layout.take(16)
        self.pool = layout.take(self.pool_stride * pool_entries) if pool_entries else 0
        # a decode step's reduction is one launch whose flags arrive in the reader's own memory (the slot layout of the
        # EXL3 layer's step); many rows (owner runs) and steps beyond that launch's size keep the two-launch form
        self.flags = not wide and rows * H <= R.ORDERED_COLLECTIVE_MAXIMUM_ELEMENTS
        self.slot_input = R.EXL3_LAYER_SIGNAL_BYTES if self.flags else SIGNAL_BYTES
        self.parity_stride = api.align(self.slot_input + rows * H * 4, LINE)
        self.region = layout.take(2 * self.parity_stride, LINE)
        self.picks = layout.take(rows * c.picks * 4)
        self.weights = layout.take(rows * c.picks * 4)
        self.jobs = layout.take(self.job_capacity * 96)
        self.expert_table = layout.take(c.experts * 24)
        # many rows: counts and entries of the grouping launch (the head of the prefill's workspace)
        self.workspace_bytes = api.prefill_parts(rows, c.picks, 0, c.experts, H, I).gate_up_operands if wide else 0
        self.workspace = layout.take(self.workspace_bytes, 1024) if wide else 0
        self.sizes = {"codes": rows * H, "exponents": rows * H // 32, "operands": rows * H * 2,
                      "hidden": pairs * I * 2, "hidden_codes": pairs * I, "hidden_exponents": pairs * I // 32,
                      "hidden_operands": pairs * I * 2, "pair_output": pairs * H * 2, "row_output": rows * H * 4}
        self.at = {name: layout.take(size) for name, size in self.sizes.items()}
        self.shared_sizes = {"gate_output": rows * I * 2, "up_output": rows * I * 2, "hidden": rows * I * 2,
                             "hidden_codes": rows * I, "hidden_exponents": rows * I // 32,
                             "hidden_operands": rows * I * 2, "output": rows * H * 2} if c.shared else {}
        # the tensor-core products' vectors: codes in stream order; for many rows tiles of 128 vectors in operand order
        self.stream_codes = layout.take(rows * H)
        tiles = 0
        if wide and tensor_products(config, I, True, True):
            tiles = api.prefill_parts(rows, c.picks, 0, c.experts, H, I).tile_capacity + (rows + 31) // 32
        self.tile_sizes = {"codes": tiles * 128 * H, "exponents": tiles * 4 * H, "hidden_codes": tiles * 128 * I,
                           "hidden_exponents": tiles * 4 * I}
        self.tile_at = {name: layout.take(size, 1024) for name, size in self.tile_sizes.items()}
        self.shared_at = {name: layout.take(size) for name, size in self.shared_sizes.items()}
        self.weights_begin = api.align(layout.cursor, 64)
        self.matrices = []
        for _ in range(c.experts):
            self.matrices.append((layout.take(matrix_bytes(I, H), 64), layout.take(matrix_bytes(I, H), 64),
                                  layout.take(matrix_bytes(H, I), 64)))
        self.weights_end = layout.cursor
        self.shared_matrices = (layout.take(shared_matrix_bytes(I, H, block128), 64),
                                layout.take(shared_matrix_bytes(I, H, block128), 64),
                                layout.take(shared_matrix_bytes(H, I, block128), 64)) if c.shared else ()
        self.arena_bytes = api.align(layout.cursor, 4096) + 4096


class MxLayer:
    def __init__(self, card, config, matrices, rank=0, rank_count=1, slices=(4, 4), shared_matrices=None,
                 shared_slices=(2, 2), pool_entries=0, block128=False, wide=False, many=True, side_run=True):
        """matrices: iterable over the routed experts of this rank's (gate, up, down) stored MXFP4 bytes;
        shared_matrices: the always-on expert's (gate, up, down) stored E4M3 bytes, where the configuration has one:
        WEIGHT_FORMAT_E4M3_SCALED, or with block128 WEIGHT_FORMAT_E4M3_BLOCK128 (one FP32 scale per 128 by 128).
        slices, shared_slices, side_run: of the mma.sync launches alone (where tensor_products says so, the tensor cores
        sum all of K and the always-on expert stands in the same launches, and these say nothing): the chains a sum over K
        is cut in, of the routed and of the always-on expert; the always-on expert's launches as a side run of the step's
        graph, beside the routed experts' (the same values either way: the two touch disjoint ranges until the launch that
        joins them)."""
        self.card, self.config = card, config
        self.layout = L = MxLayout(config, rank_count, rank, pool_entries, block128, wide)
        assert card.arena_bytes >= L.arena_bytes
        self.rank, self.rank_count = rank, rank_count
        self.weight_bytes = 0
        table = np.zeros((config.experts, 3), dtype=np.uint64)
        for expert, triple in enumerate(matrices):
            for which, data in enumerate(triple):
                card.upload(L.matrices[expert][which], data)
                table[expert, which] = L.matrices[expert][which]
                self.weight_bytes += data.size
        card.upload(L.expert_table, table)
        if config.shared:
            for which, data in enumerate(shared_matrices):
                assert data.size == shared_matrix_bytes(*((L.inner_local, config.hidden) if which < 2 else
                                                          (config.hidden, L.inner_local)), block128)
                card.upload(L.shared_matrices[which], data)
                self.weight_bytes += data.size
        for offset, size in ((L.peer_table, 16 * 32), (L.status, 16), (L.step, 256), (L.region, 2 * L.parity_stride)):
            card.fill(offset, 0, size)
        peers = (R.OrderedPeer * rank_count)()
        for peer in range(rank_count):
            peers[peer].region_offset = L.region
        card.upload(L.peer_table, np.frombuffer(bytes(peers), dtype=np.uint8))
        self.sequence = 0
        self.step_graph = None  # step(): the copies and the launches as one graph, captured at its first call
        self.staged = api.StepStaging(card, L, config)
        if tensor_products(config, L.inner_local, wide, many):
            self._prepare_tensor()
        else:
            self._prepare(slices, shared_slices, many, side_run)
        self._capture()

    def _shared_format(self):
        if not self.config.shared:
            return 0
        return WEIGHT_FORMAT_E4M3_BLOCK128 if self.layout.block128 else WEIGHT_FORMAT_E4M3_SCALED

    def _routing(self):
        """The record of the prefill's routing launches: every routed expert local, no always-on expert."""
        c, L = self.config, self.layout
        routing = R.Exl3Prefill()
        routing.scores_offset, routing.expert_table_offset = L.scores, L.expert_table
        routing.picks_offset, routing.weights_offset, routing.workspace_offset = L.picks, L.weights, L.workspace
        routing.step_offset, routing.input_size, routing.inner_size = L.step, c.hidden, L.inner_local
        routing.expert_count, routing.local_count, routing.picks = c.experts, c.experts, c.picks
        routing.row_capacity, routing.scoring, routing.route_scale = c.row_capacity, c.scoring, c.route_scale
        return routing

    def _router(self):
        c, L = self.config, self.layout
        return R.RouterSelectB200(L.scores, L.expert_table, L.picks, L.weights, L.jobs, L.step, c.experts, 0, c.picks,
                                  c.row_capacity, L.job_capacity, c.scoring, c.route_scale, 0)

    def _prepare_tensor(self):
        c, L, card, lib = self.config, self.layout, self.card, api.library()
        H, I, rows = c.hidden, L.inner_local, c.row_capacity

        def prepare(name, record, count):
            entry = getattr(lib, name)
            entry.argtypes = [C.c_void_p, C.c_uint64, C.POINTER(api.BackendOperations), C.c_void_p,
                              C.POINTER(R.KernelLaunch)]
            launches = (R.KernelLaunch * count)()
            api.check(entry(C.byref(record), card.arena_bytes, card.ops_pointer, card.handle, launches), name)
            return list(launches)
        quantize = R.MxQuantize(R.ActivationQuantize(L.tokens, L.at["codes"], L.at["exponents"], 0, H, 0),
                                L.stream_codes, L.step, rows, 0)
        description = R.MxLayerDescription()
        description.workspace_offset, description.expert_table_offset = L.workspace, L.expert_table
        description.step_offset = L.step
        if L.wide:
            head = prepare("router_tiles_prepare", self._routing(), 3) + prepare("mx_quantize_prepare", quantize, 1)
            description.row_codes = R.LinearRange(L.stream_codes, rows * H)
            description.row_exponents = R.LinearRange(L.at["exponents"], L.sizes["exponents"])
            for name in L.tile_sizes:
                setattr(description, name, R.LinearRange(L.tile_at[name], L.tile_sizes[name]))
        else:
            head = prepare("mx_route_quantize_prepare", R.MxRouteQuantize(self._router(), quantize), 1)
            description.jobs = R.LinearRange(L.jobs, L.job_capacity * 96)
            description.codes = R.LinearRange(L.stream_codes, rows * H)
            for name in ("exponents", "hidden_codes", "hidden_exponents"):
                setattr(description, name, R.LinearRange(L.at[name], L.sizes[name]))
        description.pair_output = R.LinearRange(L.at["pair_output"], L.sizes["pair_output"])
        if c.shared:
            for name in ("hidden_codes", "hidden_exponents", "output"):
                setattr(description, "shared_" + name, R.LinearRange(L.shared_at[name], L.shared_sizes[name]))
            description.shared_weights_offset = (C.c_uint64 * 3)(*L.shared_matrices)
        description.shared_format, description.hidden_size, description.inner_size = self._shared_format(), H, I
        description.expert_count, description.picks, description.row_capacity = c.experts, c.picks, rows
        description.activation_limit = c.activation_limit
        lib.mx_products_prepare.argtypes = [C.POINTER(R.MxLayerDescription), C.c_uint64,
                                            C.POINTER(api.BackendOperations), C.c_void_p, C.POINTER(R.KernelLaunch),
                                            C.POINTER(C.c_uint32)]
        launches, count = (R.KernelLaunch * 3)(), C.c_uint32()
        api.check(lib.mx_products_prepare(C.byref(description), card.arena_bytes, card.ops_pointer, card.handle, launches,
                                          C.byref(count)), "mx_products_prepare")
        self.expert_launches = list(launches)[count.value - 2:count.value]  # gate/up, down
        head += list(launches)[:count.value - 2]
        if L.wide and self.rank_count == 1:
            # no peers: row sums, the always-on expert's rows and the rounding are one launch
            one = R.OrderedRowsOne(L.at["pair_output"], 0, L.shared_at["output"] if c.shared else 0, L.at["row_output"],
                                   L.result, L.step, H, c.picks, rows, 0, 0, 0, 1, 0)
            self.launches = head + self.expert_launches + [api.rows_one(card, one)]
            return
        behind = [] if L.flags else self._row_sums()
        reduce_launches = self._reduce()
        if L.flags:
            reduce_launches[0].branch = R.LAUNCH_CHAIN | R.LAUNCH_OVERLAPS_PREVIOUS
        self.launches = head + self.expert_launches + behind + reduce_launches

    def _row_sums(self):
        """FP32 sums of the routed pairs' bfloat16 outputs, and the always-on expert's rows added to them"""
        c, L, card = self.config, self.layout, self.card
        record = R.ExpertRowSum(L.at["pair_output"], L.at["row_output"], c.hidden, c.picks)
        launch = R.KernelLaunch()
        launch.kernel = card.kernel("kernel_expert_linear", "expert_row_sum_entry", C.sizeof(record))
        launch.argument_byte_count = C.sizeof(record)
        launch.grid[:] = ((c.hidden + 255) // 256, c.row_capacity, 1)
        launch.block[:] = (256, 1, 1)
        C.memmove(launch.argument, C.byref(record), C.sizeof(record))
        return [launch] + ([self._rows_add()] if c.shared else [])

    def _rows_add(self):
        c, L, card, lib = self.config, self.layout, self.card, api.library()
        lib.linear_rows_add_prepare.argtypes = [C.POINTER(R.LinearRange), C.POINTER(R.LinearRange), C.c_uint32,
                                                C.c_uint32, C.c_uint64, C.POINTER(api.BackendOperations),
                                                C.c_void_p, C.POINTER(R.KernelLaunch)]
        add = R.KernelLaunch()
        sums = R.LinearRange(L.at["row_output"], L.sizes["row_output"])
        values = R.LinearRange(L.shared_at["output"], L.shared_sizes["output"])
        api.check(lib.linear_rows_add_prepare(C.byref(sums), C.byref(values), c.hidden, c.row_capacity, card.arena_bytes,
                                              card.ops_pointer, card.handle, C.byref(add)), "linear_rows_add_prepare")
        return add

    def _reduce(self):
        """The reduction's launches: of the pair outputs and the always-on rows in one, or of the rows' sums in two"""
        c, L, card, lib, H = self.config, self.layout, self.card, api.library(), self.config.hidden
        reduce = R.OrderedReduceBf16Description()
        reduce.reduce.collective = R.OrderedCollective(L.peer_table, L.region, L.slot_input, L.result, 0, L.step,
                                                       L.parity_stride, c.deadline_cycles, c.row_capacity * H,
                                                       self.rank_count, self.rank, 0)
        reduce.reduce.status_offset, reduce.reduce.width = L.status, H
        reduce.reduce.mode = R.ORDERED_REDUCE_OWNER_RUNS if L.wide else R.ORDERED_REDUCE_EVERY_RANK
        reduce.pair_output_offset, reduce.arena_byte_count = L.at["row_output"], card.arena_bytes
        reduce.pairs_per_row, reduce.row_capacity = 1, c.row_capacity
        lib.ordered_reduce_bf16_prepare.argtypes = [C.POINTER(R.OrderedReduceBf16Description),
                                                    C.POINTER(api.BackendOperations), C.c_void_p,
                                                    C.POINTER(R.KernelLaunch)]
        lib.ordered_publish_reduce_bf16_prepare.argtypes = [C.POINTER(R.OrderedReduceBf16Description), C.c_uint64,
                                                            C.c_uint64, C.POINTER(api.BackendOperations), C.c_void_p,
                                                            C.POINTER(R.KernelLaunch)]
        if L.flags:
            # row sums of the pair outputs, the always-on expert's rows, READY and the ranks' sum in one launch: it
            # stands for expert_row_sum_entry, trunk_rows_add_entry and the reduction's two
            reduce.pair_output_offset, reduce.pairs_per_row = L.at["pair_output"], c.picks
            reduce_launches = (R.KernelLaunch * 1)()
            api.check(lib.ordered_publish_reduce_bf16_prepare(
                C.byref(reduce), L.shared_at["output"] if c.shared else 0, L.at["row_output"], card.ops_pointer,
                card.handle, reduce_launches), "ordered_publish_reduce_bf16_prepare")
        else:
            reduce_launches = (R.KernelLaunch * 2)()
            api.check(lib.ordered_reduce_bf16_prepare(C.byref(reduce), card.ops_pointer, card.handle, reduce_launches),
                      "ordered_reduce_bf16_prepare")
        return list(reduce_launches)

    def _prepare(self, slices, shared_slices, many, side_run):
        config, L, card, wide = self.config, self.layout, self.card, self.layout.wide
        c, lib, H, I = config, api.library(), config.hidden, L.inner_local
        router = self._router()
        lib.router_select_b200_prepare.argtypes = [C.POINTER(R.RouterSelectB200), C.c_uint64,
                                                   C.POINTER(api.BackendOperations), C.c_void_p,
                                                   C.POINTER(R.KernelLaunch)]
        router_launch = R.KernelLaunch()
        if wide:
            lib.router_wide_prepare.argtypes = [C.POINTER(R.RouterWide), C.c_uint64, C.POINTER(api.BackendOperations),
                                                C.c_void_p, C.POINTER(R.KernelLaunch)]
            router_launches = (R.KernelLaunch * R.ROUTER_WIDE_LAUNCHES)()
            api.check(lib.router_wide_prepare(C.byref(R.RouterWide(self._routing(), L.jobs, L.job_capacity, 0)),
                                              card.arena_bytes, card.ops_pointer, card.handle, router_launches),
                      "router_wide_prepare")
            router_launches = list(router_launches)
        else:
            api.check(lib.router_select_b200_prepare(C.byref(router), card.arena_bytes, card.ops_pointer, card.handle,
                                                     C.byref(router_launch)), "router_select_b200_prepare")
            router_launches = [router_launch]
        kernels = R.LinearKernels()
        lib.linear_kernels_prepare.argtypes = [C.POINTER(api.BackendOperations), C.c_void_p, C.c_uint32,
                                               C.POINTER(R.LinearKernels)]
        api.check(lib.linear_kernels_prepare(card.ops_pointer, card.handle, 100, C.byref(kernels)),
                  "linear_kernels_prepare")

        def span(name):
            return R.LinearRange(L.at[name], L.sizes[name])
        quantize = R.LinearQuantizeDescription(R.LinearRange(L.tokens, c.row_capacity * H * 2), span("codes"),
                                               span("exponents"), span("operands"), H, c.row_capacity)
        lib.linear_quantize_prepare.argtypes = [C.POINTER(R.LinearQuantizeDescription), C.c_uint64,
                                                C.POINTER(R.LinearKernels), C.POINTER(R.KernelLaunch)]
        quantize_launch = R.KernelLaunch()
        api.check(lib.linear_quantize_prepare(C.byref(quantize), card.arena_bytes, C.byref(kernels),
                                              C.byref(quantize_launch)), "linear_quantize_prepare")
        head = router_launches + [quantize_launch]
        if not wide:
            # a decode step begins with the router and the rows' quantization, neither of which reads the other's
            # output: one launch (block 0 routes, the others quantize)
            lib.router_select_quantize_prepare.argtypes = [C.POINTER(R.RouterSelectB200), C.POINTER(R.KernelLaunch),
                                                           C.c_uint64, C.POINTER(api.BackendOperations), C.c_void_p,
                                                           C.POINTER(R.KernelLaunch)]
            first = R.KernelLaunch()
            api.check(lib.router_select_quantize_prepare(C.byref(router), C.byref(quantize_launch), card.arena_bytes,
                                                         card.ops_pointer, card.handle, C.byref(first)),
                      "router_select_quantize_prepare")
            head = [first]
        description = R.LinearRoutedExpertsDescription()
        description.jobs = R.LinearRange(L.jobs, L.job_capacity * 96)
        description.expert_weights = R.LinearRange(L.weights_begin, L.weights_end - L.weights_begin)
        for name in L.sizes:
            setattr(description, name, span(name))
        description.gate_up_shape, description.down_shape = R.MatrixShape(I, H, 4, 0), R.MatrixShape(H, I, 4, 0)
        description.weight_format, description.job_count = WEIGHT_FORMAT_E2M1_SCALED, L.job_capacity
        description.row_count, description.pairs_per_row = c.row_capacity, c.picks
        description.activation_limit = c.activation_limit
        description.gate_up_slice_count, description.down_slice_count = slices
        lib.linear_routed_experts_prepare.argtypes = [C.POINTER(R.LinearRoutedExpertsDescription), C.c_uint64,
                                                      C.POINTER(R.LinearKernels), C.POINTER(R.KernelLaunch)]
        lib.linear_routed_experts_wide_prepare.argtypes = [C.POINTER(R.LinearRoutedExpertsDescription), C.c_uint64,
                                                           C.POINTER(R.LinearKernels),
                                                           C.POINTER(api.BackendOperations), C.c_void_p,
                                                           C.POINTER(R.KernelLaunch)]
        self.expert_launches = (R.KernelLaunch * 4)()
        if wide and many:
            api.check(lib.linear_routed_experts_wide_prepare(C.byref(description), card.arena_bytes, C.byref(kernels),
                                                             card.ops_pointer, card.handle, self.expert_launches),
                      "linear_routed_experts_wide_prepare")
        else:
            api.check(lib.linear_routed_experts_prepare(C.byref(description), card.arena_bytes, C.byref(kernels),
                                                        self.expert_launches), "linear_routed_experts_prepare")
        shared_launches = []
        if c.shared:
            shared = R.LinearSharedExpertDescription()
            for which, (name, (o, i)) in enumerate((("gate", (I, H)), ("up", (I, H)), ("down", (H, I)))):
                setattr(shared, name, R.LinearMatrix(R.LinearRange(L.shared_matrices[which],
                                                                   shared_matrix_bytes(o, i, L.block128)),
                                                     R.MatrixShape(o, i, 8, 0),
                                                     WEIGHT_FORMAT_E4M3_BLOCK128 if L.block128 else
                                                     WEIGHT_FORMAT_E4M3_SCALED,
                                                     shared_slices[0 if which < 2 else 1], 0, 0))
            shared.codes, shared.exponents, shared.operands = span("codes"), span("exponents"), span("operands")
            for name in L.shared_sizes:
                setattr(shared, name, R.LinearRange(L.shared_at[name], L.shared_sizes[name]))
            shared.row_count, shared.activation_limit = c.row_capacity, c.activation_limit
            lib.linear_shared_expert_prepare.argtypes = [C.POINTER(R.LinearSharedExpertDescription), C.c_uint64,
                                                         C.POINTER(R.LinearKernels), C.POINTER(R.KernelLaunch)]
            lib.linear_shared_expert_block128_prepare.argtypes = [C.POINTER(R.LinearSharedExpertDescription), C.c_uint64,
                                                                  C.POINTER(R.LinearKernels),
                                                                  C.POINTER(api.BackendOperations), C.c_void_p,
                                                                  C.POINTER(R.KernelLaunch)]
            lib.linear_shared_expert_wide_prepare.argtypes = lib.linear_shared_expert_block128_prepare.argtypes
            four = (R.KernelLaunch * 4)()
            if wide:
                api.check(lib.linear_shared_expert_wide_prepare(C.byref(shared), card.arena_bytes, C.byref(kernels),
                                                                card.ops_pointer, card.handle, four),
                          "linear_shared_expert_wide_prepare")
            elif L.block128:
                api.check(lib.linear_shared_expert_block128_prepare(C.byref(shared), card.arena_bytes, C.byref(kernels),
                                                                    card.ops_pointer, card.handle, four),
                          "linear_shared_expert_block128_prepare")
            else:
                api.check(lib.linear_shared_expert_prepare(C.byref(shared), card.arena_bytes, C.byref(kernels), four),
                          "linear_shared_expert_prepare")
            shared_launches = list(four) + [self._rows_add()]
        reduce_launches = self._reduce()
        self.step_launches = list(self.expert_launches)
        if L.flags:
            self.step_launches = self.step_launches[:3]
            shared_launches = shared_launches[:4]
        # the always-on expert reads the quantized rows alone: its four launches are a side run of the graph beside the
        # routed experts' launches (a decode step's trunk launches are too small to fill the card by themselves);
        # the join is the launch that adds its rows to the routed experts' sums
        behind = shared_launches[4:] + list(reduce_launches)  # the launch that joins the two runs first
        if shared_launches and side_run:
            for launch in shared_launches[:4]:
                launch.branch = R.LAUNCH_SIDE
            self.expert_launches[0].branch = R.LAUNCH_RESUME
            behind[0].branch = R.LAUNCH_JOIN
            self.launches = head + shared_launches[:4] + self.step_launches + behind
        else:
            self.launches = head + self.step_launches + shared_launches[:4] + behind

    def _capture(self):
        L, card, lib = self.layout, self.card, api.library()
        self.graph = card.graph(self.launches)
        self.resident_graph = None
        if L.pool_entries:
            select = R.StepInputSelect(L.pool, L.pool_stride, L.step, L.cursor, L.pool_entries, L.step_input_bytes)
            lib.step_input_select_prepare.argtypes = [C.POINTER(R.StepInputSelect), C.c_uint64,
                                                      C.POINTER(api.BackendOperations), C.c_void_p,
                                                      C.POINTER(R.KernelLaunch)]
            select_launch = R.KernelLaunch()
            api.check(lib.step_input_select_prepare(C.byref(select), card.arena_bytes, card.ops_pointer, card.handle,
                                                    C.byref(select_launch)), "step_input_select_prepare")
            self.resident_graph = card.graph([select_launch] + self.launches)

    def load_pool(self, steps):
        """steps: pool_entries tuples (sequence, tokens, scores), sequences strictly increasing. Their input areas go
        to the card's pool; run_resident() then takes them one after the other without touching the host."""
        L, card = self.layout, self.card
        assert len(steps) == L.pool_entries
        for index, (sequence, tokens, scores) in enumerate(steps):
            self.stage_step(0, sequence, tokens, scores)
            card.transfer_wait(card.upload_async(L.pool + index * L.pool_stride, 0, L.step_input_bytes))
        card.fill(L.cursor, 0, 16)
        card.wait()

    def run_resident(self):
        self.card.graph_run(self.resident_graph)

    def connect_local(self, layers):
        for peer, other in enumerate(layers):
            self.card.peer_connect(other.card, 0, self.layout.peer_table + 32 * peer)

    def connect_handles(self, handles):
        for peer, handle in enumerate(handles):
            if peer == self.rank:
                self.card.peer_connect(self.card, 0, self.layout.peer_table + 32 * peer)
            else:
                self.card.ipc_connect(handle, 0, self.layout.peer_table + 32 * peer)

    def stage_step(self, staging_offset, sequence, tokens, scores):
        L, view = self.layout, self.card.staging_view
        block = R.StepBlock(sequence, tokens.shape[0], 0)
        view[staging_offset:staging_offset + 16] = np.frombuffer(bytes(block), dtype=np.uint8)
        at = staging_offset + (L.tokens - L.step)
        view[at:at + tokens.nbytes] = tokens.reshape(-1).view(np.uint8)
        at = staging_offset + (L.scores - L.step)
        view[at:at + scores.nbytes] = np.ascontiguousarray(scores, dtype=np.float32).reshape(-1).view(np.uint8)

    def submit(self, staging_offset, result_staging_offset, rows):
        L, card = self.layout, self.card
        card.upload_async(L.step, staging_offset, L.step_input_bytes)
        card.graph_run(self.graph)
        return card.download_async(L.result, result_staging_offset, rows * self.config.hidden * 2)

    def step(self, tokens, scores):
        """One layer call on host arrays; returns bfloat16 bits [rows][hidden]. Raises if a kernel of it gave up a wait."""
        L, card = self.layout, self.card
        self.sequence += 1
        if L.wide:
            # one library call on ordinary memory: a prompt's rows in, the graph, status block and result out, wait
            rows = tokens.shape[0]
            status, result = np.empty(4, np.uint32), np.empty((rows, self.config.hidden), np.uint16)
            block = np.array([self.sequence, rows], dtype=np.uint64)
            card.call(self.graph, [(L.step, block), (L.tokens, np.ascontiguousarray(tokens)),
                                   (L.scores, np.ascontiguousarray(scores, dtype=np.float32))],
                      [(L.status, status), (L.result, result)])
            self._raise_on(status)
            return result
        status, result = self.staged.write(self.sequence, tokens, scores)
        result_at = self.staged.result_at
        # one library call: inputs in, the graph, status block and result out, wait. The copies are nodes of the step's
        # own graph where its table is a plain chain
        if self.step_graph is None:
            captured = card.step_capture(self.launches, L.step, 0, L.step_input_bytes, L.status, result_at,
                                         16 + self.config.row_capacity * self.config.hidden * 2)
            self.step_graph = -1 if captured is None else captured
        if self.step_graph >= 0:
            card.graph_run_wait(self.step_graph)
        else:
            card.step_run(self.graph, L.step, 0, L.step_input_bytes, L.status, result_at, 16 + result.nbytes)
        self._raise_on(status)
        return result.copy()

    def check_status(self):
        """What step raises, of the steps that were submitted (it waits for them)."""
        self.card.check_waits()
        self._raise_on(self.card.download(self.layout.status, 16, np.uint32))

    @staticmethod
    def _raise_on(status):
        if status[0] != 0:
            raise RuntimeError("ordered reduction failed: code %d (1 timed out, 2 bad sequence), phase %d, rank %d"
                               % (status[0], status[1], status[2]))
