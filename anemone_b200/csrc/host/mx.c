/*
 * mx.c: preparation of the original-weights layer's tensor-core launches (anemone_b200_mx.h).
 */
#include "anemone_b200_mx.h"

#include <math.h>
#include <string.h>

#include "prepare_common.h"

#define MX_WIDTH_STEP 128u /* a block of the products' inputs; a unit of down's outputs */
#define MX_SMS 148u /* one persistent CTA a SM */

static bool range_holds(const struct linear_range *range, uint64_t needed)
{
	return needed != UINT64_MAX && range->byte_count >= needed;
}

static result_status one_kernel(const struct backend_operations *backend, struct device_card *card, const char *file,
				const char *name, uint32_t record_bytes, uint32_t *kernel_out)
{
	*kernel_out = BACKEND_NO_KERNEL;
	const result_status status = backend->kernel_prepare(card, file, name, record_bytes, kernel_out);
	return status == STATUS_OK && *kernel_out == BACKEND_NO_KERNEL ? STATUS_UNSUPPORTED : status;
}

static bool quantize_is_valid(const struct mx_quantize_arguments *arguments, uint64_t arena_byte_count)
{
	const uint64_t rows = arguments->row_capacity, width = arguments->base.width;
	const struct checked_range ranges[5] = {
		{ "values", arguments->base.values_offset, linear_values_byte_count(rows, (uint32_t)width) },
		{ "codes", arguments->base.codes_offset, linear_codes_byte_count(rows, (uint32_t)width) },
		{ "exponents", arguments->base.exponents_offset, linear_exponents_byte_count(rows, (uint32_t)width) },
		{ "stream codes", arguments->stream_offset, linear_codes_byte_count(rows, (uint32_t)width) },
		{ "step block", arguments->step_offset, sizeof(struct step_block) }
	};
	return arguments->reserved_zero == 0 && arguments->base.reserved_zero == 0 && rows != 0 && width != 0 &&
	       width % LINEAR_VALUES_PER_LOAD == 0 && prepare_ranges_are_valid("mx quantize", ranges, 5, arena_byte_count);
}

result_status mx_quantize_prepare(const struct mx_quantize_arguments *arguments, uint64_t arena_byte_count,
				  const struct backend_operations *backend, struct device_card *card,
				  struct kernel_launch *launch_out)
{
	if (arguments == NULL || backend == NULL || backend->kernel_prepare == NULL || card == NULL || launch_out == NULL ||
	    !quantize_is_valid(arguments, arena_byte_count))
		return STATUS_INVALID_ARGUMENT;
	uint32_t kernel;
	const result_status status =
		one_kernel(backend, card, MX_KERNEL_FILE, "mx_quantize", sizeof(*arguments), &kernel);
	if (status != STATUS_OK)
		return status;
	/* a warp a load, eight warps a block; the blocks a card holds at once walk the rest */
	const uint64_t blocks = ((uint64_t)arguments->row_capacity * (arguments->base.width / LINEAR_VALUES_PER_LOAD) + 7u) / 8u;
	prepare_launch_fill(launch_out, kernel, (uint32_t)(blocks < 8u * MX_SMS ? blocks : 8u * MX_SMS), 1, 1, 256, 0,
			    arguments, sizeof(*arguments));
	return STATUS_OK;
}

result_status mx_route_quantize_prepare(const struct mx_route_quantize_arguments *arguments, uint64_t arena_byte_count,
					const struct backend_operations *backend, struct device_card *card,
					struct kernel_launch *launch_out)
{
	struct kernel_launch checked;
	if (arguments == NULL || launch_out == NULL)
		return STATUS_INVALID_ARGUMENT;
	const result_status valid =
		router_select_b200_prepare(&arguments->router, arena_byte_count, backend, card, &checked);
	if (valid != STATUS_OK)
		return valid;
	if (!quantize_is_valid(&arguments->quantize, arena_byte_count))
		return STATUS_INVALID_ARGUMENT;
	uint32_t kernel;
	const result_status status = one_kernel(backend, card, KERNEL_FILE_ROUTER_B200, "mx_route_quantize",
						sizeof(*arguments), &kernel);
	if (status != STATUS_OK)
		return status;
	/* block 0 routes; a warp of the others takes a load of 64 values */
	const uint32_t warps = ROUTER_B200_THREADS / 32u;
	const uint64_t tasks = (uint64_t)arguments->quantize.row_capacity *
			       (arguments->quantize.base.width / LINEAR_VALUES_PER_LOAD);
	const uint64_t blocks = (tasks + warps - 1u) / warps;
	prepare_launch_fill(launch_out, kernel, 1u + (uint32_t)(blocks < MX_SMS ? blocks : MX_SMS), 1, 1,
			    ROUTER_B200_THREADS, 0, arguments, sizeof(*arguments));
	launch_out->branch = LAUNCH_CHAIN | LAUNCH_OVERLAPS_PREVIOUS; /* behind the copy of the step's inputs */
	return STATUS_OK;
}

result_status router_tiles_prepare(const struct exl3_prefill_record *routing, uint64_t arena_byte_count,
				   const struct backend_operations *backend, struct device_card *card,
				   struct kernel_launch *launches_out)
{
	if (routing == NULL || backend == NULL || backend->kernel_prepare == NULL || card == NULL || launches_out == NULL)
		return STATUS_INVALID_ARGUMENT;
	const uint64_t rows = routing->row_capacity;
	if (routing->expert_count == 0 || routing->expert_count > ROUTER_B200_MAXIMUM_EXPERTS || routing->local_first != 0 ||
	    routing->local_count != routing->expert_count || routing->shared_count != 0 || routing->picks == 0 ||
	    routing->picks > ROUTER_B200_MAXIMUM_PICKS || routing->picks > routing->expert_count || rows == 0 ||
	    rows > 65535u || routing->scoring > ROUTER_SCORING_SQRT_SOFTPLUS || !isfinite(routing->route_scale) ||
	    routing->route_scale <= 0 || routing->workspace_offset % 1024u != 0)
		return STATUS_INVALID_ARGUMENT;
	const struct exl3_prefill_parts parts = exl3_prefill_parts_of(routing->row_capacity, routing->picks, 0,
								      routing->expert_count, routing->input_size,
								      routing->inner_size);
	const struct checked_range ranges[6] = {
		{ "bias", routing->bias_offset, routing->bias_offset != 0 ? (uint64_t)routing->expert_count * 4u : 0u },
		{ "scores", routing->scores_offset, rows * routing->expert_count * 4u },
		{ "picks", routing->picks_offset, rows * routing->picks * 4u },
		{ "weights", routing->weights_offset, rows * routing->picks * 4u },
		{ "workspace", routing->workspace_offset, parts.gate_up_operands },
		{ "step block", routing->step_offset, sizeof(struct step_block) }
	};
	if (!prepare_ranges_are_valid("router tiles", ranges, 6, arena_byte_count))
		return STATUS_INVALID_ARGUMENT;
	const uint32_t row_warps = ROUTER_B200_THREADS / 32u;
	const struct {
		const char *name;
		uint32_t blocks, threads;
	} shapes[ROUTER_TILES_LAUNCHES] = {
		{ "exl3_prefill_picks", (routing->row_capacity + row_warps - 1u) / row_warps, ROUTER_B200_THREADS },
		{ "exl3_prefill_group", routing->expert_count, 256u },
		{ "exl3_prefill_tiles", 1u, ROUTER_B200_THREADS }
	};
	struct kernel_launch launches[ROUTER_TILES_LAUNCHES];
	for (uint32_t index = 0; index < ROUTER_TILES_LAUNCHES; index++) {
		uint32_t kernel;
		const result_status status = one_kernel(backend, card, EXL3_PREFILL_KERNEL_FILE, shapes[index].name,
							sizeof(*routing), &kernel);
		if (status != STATUS_OK)
			return status;
		prepare_launch_fill(&launches[index], kernel, shapes[index].blocks, 1, 1, shapes[index].threads, 0, routing,
				    sizeof(*routing));
	}
	memcpy(launches_out, launches, sizeof(launches));
	return STATUS_OK;
}

result_status mx_products_prepare(const struct mx_layer_description *description, uint64_t arena_byte_count,
				  const struct backend_operations *backend, struct device_card *card,
				  struct kernel_launch launches_out[MX_PRODUCTS_LAUNCHES], uint32_t *launch_count_out)
{
	if (description == NULL || backend == NULL || backend->kernel_prepare == NULL || card == NULL || launches_out == NULL ||
	    launch_count_out == NULL || description->reserved_zero != 0)
		return STATUS_INVALID_ARGUMENT;
	const struct mx_layer_description *const d = description;
	const uint32_t H = d->hidden_size, I = d->inner_size;
	const uint64_t rows = d->row_capacity, pairs = rows * d->picks;
	const bool shared = d->shared_format != MX_SHARED_NONE, few = d->jobs.byte_count != 0;
	if (H == 0 || H % MX_WIDTH_STEP != 0 || I == 0 || I % MX_WIDTH_STEP != 0 || d->expert_count == 0 ||
	    d->expert_count > ROUTER_B200_MAXIMUM_EXPERTS || d->picks == 0 || d->picks > ROUTER_B200_MAXIMUM_PICKS ||
	    rows == 0 || rows > 65535u || (shared && d->shared_format != WEIGHT_FORMAT_E4M3_SCALED &&
					   d->shared_format != WEIGHT_FORMAT_E4M3_BLOCK128) ||
	    (few && shared && rows > LINEAR_MAXIMUM_ROWS) || !isfinite(d->activation_limit) || d->activation_limit <= 0)
		return STATUS_INVALID_ARGUMENT;
	const struct exl3_prefill_parts parts =
		exl3_prefill_parts_of(d->row_capacity, d->picks, 0, d->expert_count, H, I);
	const uint64_t tiles = few ? d->jobs.byte_count / sizeof(struct expert_job_record) : parts.tile_capacity;
	const uint64_t all_tiles = mx_tile_count(d->row_capacity, d->picks, d->expert_count);
	/* vectors a range of codes holds: rows and pairs, or whole tiles */
	const uint64_t in = few ? rows : all_tiles * MX_TILE_ROWS, hidden = few ? pairs : all_tiles * MX_TILE_ROWS;
	if (tiles == 0 || (tiles + rows) > UINT32_MAX / (H / 64u + I / 64u) ||
	    !range_holds(&d->codes, linear_codes_byte_count(in, H)) ||
	    !range_holds(&d->exponents, linear_exponents_byte_count(in, H)) ||
	    !range_holds(&d->hidden_codes, linear_codes_byte_count(hidden, I)) ||
	    !range_holds(&d->hidden_exponents, linear_exponents_byte_count(hidden, I)) ||
	    !range_holds(&d->pair_output, linear_values_byte_count(pairs, H)) ||
	    (!few && (!range_holds(&d->row_codes, linear_codes_byte_count(rows, H)) ||
		      !range_holds(&d->row_exponents, linear_exponents_byte_count(rows, H)))) ||
	    (few && shared && (!range_holds(&d->shared_hidden_codes, linear_codes_byte_count(rows, I)) ||
			       !range_holds(&d->shared_hidden_exponents, linear_exponents_byte_count(rows, I)))) ||
	    (shared && !range_holds(&d->shared_output, linear_values_byte_count(rows, H))))
		return STATUS_INVALID_ARGUMENT;
	/* stored bytes of an always-on matrix: widths are multiples of 128, so the three matrices' are the same */
	const uint64_t matrix = !shared ? 0u :
				d->shared_format == WEIGHT_FORMAT_E4M3_BLOCK128 ?
					  (uint64_t)H * I + (uint64_t)(H / 128u) * (I / 128u) * 4u :
					  e4m3_scaled_byte_count(I, H);
	const bool few_shared = few && shared;
	const struct checked_range ranges[17] = {
		{ "jobs", d->jobs.byte_offset, d->jobs.byte_count },
		{ "workspace", few ? 0u : d->workspace_offset, few ? 0u : parts.gate_up_operands },
		{ "expert table", d->expert_table_offset, (uint64_t)d->expert_count * 24u },
		{ "step block", d->step_offset, sizeof(struct step_block) },
		{ "row codes", few ? 0u : d->row_codes.byte_offset, few ? 0u : d->row_codes.byte_count },
		{ "row exponents", few ? 0u : d->row_exponents.byte_offset, few ? 0u : d->row_exponents.byte_count },
		{ "codes", d->codes.byte_offset, d->codes.byte_count },
		{ "exponents", d->exponents.byte_offset, d->exponents.byte_count },
		{ "hidden codes", d->hidden_codes.byte_offset, d->hidden_codes.byte_count },
		{ "hidden exponents", d->hidden_exponents.byte_offset, d->hidden_exponents.byte_count },
		{ "pair output", d->pair_output.byte_offset, d->pair_output.byte_count },
		{ "always-on hidden codes", few_shared ? d->shared_hidden_codes.byte_offset : 0u,
		  few_shared ? d->shared_hidden_codes.byte_count : 0u },
		{ "always-on hidden exponents", few_shared ? d->shared_hidden_exponents.byte_offset : 0u,
		  few_shared ? d->shared_hidden_exponents.byte_count : 0u },
		{ "always-on output", shared ? d->shared_output.byte_offset : 0u, shared ? d->shared_output.byte_count : 0u },
		{ "always-on gate", shared ? d->shared_weights_offset[0] : 0u, matrix },
		{ "always-on up", shared ? d->shared_weights_offset[1] : 0u, matrix },
		{ "always-on down", shared ? d->shared_weights_offset[2] : 0u, matrix }
	};
	if (!prepare_ranges_are_valid("mx products", ranges, 17, arena_byte_count))
		return STATUS_INVALID_ARGUMENT;
	struct mx_products_arguments gate_up;
	memset(&gate_up, 0, sizeof(gate_up));
	gate_up.jobs_offset = few ? d->jobs.byte_offset : 0u;
	gate_up.counts_offset = few ? 0u : d->workspace_offset + parts.counts;
	gate_up.tiles_offset = few ? 0u : d->workspace_offset + parts.tiles;
	gate_up.entries_offset = few ? 0u : d->workspace_offset + parts.entries;
	gate_up.expert_table_offset = d->expert_table_offset;
	gate_up.step_offset = d->step_offset;
	gate_up.pairs_per_row = d->picks;
	gate_up.row_capacity = d->row_capacity;
	gate_up.tile_capacity = (uint32_t)tiles;
	gate_up.expert_count = d->expert_count;
	gate_up.shared_format = d->shared_format;
	gate_up.activation_limit = d->activation_limit;
	struct mx_products_arguments down = gate_up;
	gate_up.codes_offset = gate_up.shared_codes_offset = d->codes.byte_offset;
	gate_up.exponents_offset = gate_up.shared_exponents_offset = d->exponents.byte_offset;
	gate_up.output_offset = down.codes_offset = d->hidden_codes.byte_offset;
	gate_up.output_exponents_offset = down.exponents_offset = d->hidden_exponents.byte_offset;
	down.output_offset = d->pair_output.byte_offset;
	if (shared) {
		gate_up.shared_weights_offset[0] = d->shared_weights_offset[0];
		gate_up.shared_weights_offset[1] = d->shared_weights_offset[1];
		gate_up.shared_output_offset = down.shared_codes_offset = d->shared_hidden_codes.byte_offset;
		gate_up.shared_output_exponents_offset = down.shared_exponents_offset = d->shared_hidden_exponents.byte_offset;
		down.shared_weights_offset[0] = down.shared_weights_offset[1] = d->shared_weights_offset[2];
		down.shared_output_offset = d->shared_output.byte_offset;
	}
	gate_up.input_size = down.output_size = H;
	gate_up.output_size = down.input_size = I;
	const uint64_t shared_rows = mx_shared_tile_rows(d->shared_format);
	const uint64_t shared_tiles = shared ? (rows + shared_rows - 1u) / shared_rows : 0u;
	const struct mx_gather_arguments gather = { .codes_offset = d->row_codes.byte_offset,
						    .exponents_offset = d->row_exponents.byte_offset,
						    .tile_codes_offset = d->codes.byte_offset,
						    .tile_exponents_offset = d->exponents.byte_offset,
						    .counts_offset = gate_up.counts_offset,
						    .tiles_offset = gate_up.tiles_offset,
						    .entries_offset = gate_up.entries_offset,
						    .step_offset = d->step_offset,
						    .width = H,
						    .pairs_per_row = d->picks,
						    .row_capacity = d->row_capacity,
						    .tile_capacity = (uint32_t)tiles,
						    .expert_count = d->expert_count,
						    .shared_format = d->shared_format };
	const struct {
		const char *name;
		const void *record;
		uint32_t bytes, x, y, threads, shared, branch;
	} shapes[MX_PRODUCTS_LAUNCHES] = {
		{ "mx_gather", &gather, sizeof(gather), (uint32_t)(tiles + shared_tiles), (H + 511u) / 512u, 256u, 0u,
		  LAUNCH_CHAIN },
		/* the products may each take their places on the card while the launch before them still runs */
		{ few ? "mx_gate_up_few" : "mx_gate_up_many", &gate_up, sizeof(gate_up), MX_SMS, 1u, MX_PRODUCTS_THREADS,
		  MX_PRODUCTS_DYNAMIC_BYTES, LAUNCH_CHAIN | LAUNCH_OVERLAPS_PREVIOUS },
		{ few ? "mx_down_few" : "mx_down_many", &down, sizeof(down), MX_SMS, 1u, MX_PRODUCTS_THREADS,
		  MX_PRODUCTS_DYNAMIC_BYTES, LAUNCH_CHAIN | LAUNCH_OVERLAPS_PREVIOUS }
	};
	struct kernel_launch launches[MX_PRODUCTS_LAUNCHES];
	uint32_t count = 0;
	for (uint32_t index = few ? 1u : 0u; index < MX_PRODUCTS_LAUNCHES; index++) {
		uint32_t kernel;
		const result_status status =
			one_kernel(backend, card, MX_KERNEL_FILE, shapes[index].name, shapes[index].bytes, &kernel);
		if (status != STATUS_OK)
			return status;
		prepare_launch_fill(&launches[count], kernel, shapes[index].x, shapes[index].y, 1, shapes[index].threads,
				    shapes[index].shared, shapes[index].record, shapes[index].bytes);
		launches[count++].branch = shapes[index].branch;
	}
	memcpy(launches_out, launches, count * sizeof(launches[0]));
	*launch_count_out = count;
	return STATUS_OK;
}
