/*
 * anemone_b200_mx.h: the original-weights layer's products on the fifth-generation tensor cores (B200 extension; the
 * reference's counterparts are its mma.sync expert and trunk kernels, source/kernel_expert_linear.cu and
 * source/kernel_trunk_linear.cu). Two product launches take every routed expert (MXFP4) and the always-on expert
 * (E4M3, either scale format) of a step or of a prompt; formats, arrays and the hidden step are those of
 * anemone_b200_records.h. What differs from the mma.sync launches: the FP32 sums over a vector's inputs are the tensor
 * cores' (block-scaled products accumulated in tensor memory) instead of one chain a slice, and the hidden vectors
 * are quantized where they are made.
 */
#ifndef ANEMONE_B200_MX_H
#define ANEMONE_B200_MX_H

#include "anemone_b200_backend.h"
#include "anemone_b200_linear.h"
#include "anemone_b200_records.h"
#include "anemone_b200_router.h"

#ifdef __cplusplus
extern "C" {
#endif

/* STREAM ORDER of a vector's E4M3 codes: byte 64 l + 32 q + 8 t + 2 j + p of a vector is the code of its value
 * 64 l + 32 q + 16 p + 2 t + j / 2 + 8 (j % 2). A block of 32 values stays together, and the sixteen bytes a tensor-core
 * operand row takes at a time are contiguous; within a block the order is that in which the lane order of the stored
 * weights unpacks. */
#define MX_KERNEL_FILE "kernel_mx_tensor"
#define MX_TILE_ROWS 128u /* most rows of one expert a unit multiplies */
#define MX_SHARED_NONE 0u
#define MX_BLOCK128_ROWS 32u /* most rows of a unit whose sums an epilogue lane keeps in registers */
#define MX_PRODUCTS_THREADS 896u
#define MX_PRODUCTS_DYNAMIC_BYTES 221184u

/* rows of one tile of the always-on expert */
AB_INLINE uint32_t mx_shared_tile_rows(uint32_t shared_format)
{
	return shared_format == WEIGHT_FORMAT_E4M3_BLOCK128 ? MX_BLOCK128_ROWS : MX_TILE_ROWS;
}

/* mx_quantize: grid (blocks) x 256: activation_quantize_entry's codes (lane order) and exponents of the live rows, and
 * their codes in stream order; no operands. */
struct mx_quantize_arguments {
	struct activation_quantize_arguments base; /* operands_offset unused */
	uint64_t stream_offset; /* written: codes in stream order [row_capacity][width] */
	uint64_t step_offset; /* struct step_block: row_count live rows */
	uint32_t row_capacity;
	uint32_t reserved_zero;
};

/* mx_route_quantize (kernel file kernel_router_b200): router_select_b200 and mx_quantize of a decode step in one launch */
struct mx_route_quantize_arguments {
	struct router_select_b200_arguments router;
	struct mx_quantize_arguments quantize;
};

/* OPERAND ORDER of a tile of 128 vectors: codes: the sixteen stream-order bytes 16 c .. 16 c + 15 of vector r at byte
 * 2048 c + 16 r of the tile (128 x width bytes); exponents: the four codes of 128 values' block b of vector r at byte
 * 512 b + 16 (r % 32) + 4 (r / 32) (4 x width bytes). Vectors a tile does not have are not written. */
/* mx_gather: grid (tiles, ceil(width / 512)) x 256: the rows of the routed tiles, then of the always-on expert's, in
 * operand order */
struct mx_gather_arguments {
	uint64_t codes_offset; /* stream order [row_capacity][width] */
	uint64_t exponents_offset;
	uint64_t tile_codes_offset; /* written */
	uint64_t tile_exponents_offset; /* written */
	uint64_t counts_offset; /* uint32 [expert_count + 1], the last: tile count */
	uint64_t tiles_offset;
	uint64_t entries_offset;
	uint64_t step_offset;
	uint32_t width;
	uint32_t pairs_per_row;
	uint32_t row_capacity;
	uint32_t tile_capacity;
	uint32_t expert_count;
	uint32_t shared_format;
};

/* mx_gate_up_few / mx_down_few, mx_gate_up_many / mx_down_many: a persistent grid over units: (tile of rows of one
 * expert) x (64 columns of gate and of up, or 128 outputs of down). FEW: a tile is a job of a job table, vectors are
 * stored by row and by pair. MANY: tiles are the grouping launches' (counts, tiles, entries; struct exl3_prefill_tile)
 * and, behind the tile capacity, runs of rows for the always-on expert; vectors are in operand order. */
struct mx_products_arguments {
	uint64_t jobs_offset; /* FEW: struct expert_job_record [tile_capacity] */
	uint64_t counts_offset; /* MANY */
	uint64_t tiles_offset;
	uint64_t entries_offset;
	uint64_t expert_table_offset; /* uint64 [expert_count][3] */
	uint64_t step_offset;
	uint64_t codes_offset; /* FEW: gate/up [row][input_size], down [pair][input_size]; MANY: [tile] */
	uint64_t exponents_offset;
	uint64_t shared_codes_offset; /* FEW: the always-on expert's vectors, a row each */
	uint64_t shared_exponents_offset;
	uint64_t shared_weights_offset[2]; /* gate and up, or down */
	uint64_t output_offset; /* gate/up: hidden codes, as the down launch reads them; down: bfloat16 [pair][output_size] */
	uint64_t output_exponents_offset; /* gate/up alone */
	uint64_t shared_output_offset; /* FEW gate/up and down: the same by row */
	uint64_t shared_output_exponents_offset;
	uint32_t input_size;
	uint32_t output_size;
	uint32_t pairs_per_row;
	uint32_t row_capacity;
	uint32_t tile_capacity;
	uint32_t expert_count;
	uint32_t shared_format; /* MX_SHARED_NONE, WEIGHT_FORMAT_E4M3_SCALED or WEIGHT_FORMAT_E4M3_BLOCK128 */
	float activation_limit;
};

/* The layer's arrays; widths are multiples of 128. FEW: jobs is a job table of at most eight rows a job, and the vectors'
 * ranges are by row, by pair and (shared_*) by row. MANY: jobs.byte_count is 0, workspace_offset is router_tiles_prepare's,
 * codes and hidden_codes are mx_tile_count tiles in operand order and row_codes, row_exponents the rows mx_gather reads. */
struct mx_layer_description {
	struct linear_range jobs;
	uint64_t workspace_offset;
	uint64_t expert_table_offset;
	uint64_t step_offset;
	struct linear_range row_codes; /* MANY: stream order [row_capacity][hidden_size] */
	struct linear_range row_exponents;
	struct linear_range codes; /* FEW: stream order [row_capacity][hidden_size]; MANY: scratch, tiles */
	struct linear_range exponents;
	struct linear_range hidden_codes; /* scratch: FEW [pairs][inner_size]; MANY: tiles */
	struct linear_range hidden_exponents;
	struct linear_range pair_output; /* written: bfloat16 [pairs][hidden_size] */
	struct linear_range shared_hidden_codes; /* FEW: scratch [row_capacity][inner_size] */
	struct linear_range shared_hidden_exponents;
	struct linear_range shared_output; /* written: bfloat16 [row_capacity][hidden_size] */
	uint64_t shared_weights_offset[3]; /* gate, up, down */
	uint32_t shared_format; /* MX_SHARED_NONE or the three matrices' weight format */
	uint32_t hidden_size;
	uint32_t inner_size;
	uint32_t expert_count;
	uint32_t picks;
	uint32_t row_capacity;
	float activation_limit;
	uint32_t reserved_zero;
};

/* tiles (of 128 vectors' room) of the MANY form: the routed experts' and, in either format, the always-on expert's */
AB_INLINE uint32_t mx_tile_count(uint32_t row_capacity, uint32_t picks, uint32_t expert_count)
{
	return exl3_prefill_parts_of(row_capacity, picks, 0u, expert_count, 128u, 128u).tile_capacity +
	       (row_capacity + MX_BLOCK128_ROWS - 1u) / MX_BLOCK128_ROWS;
}

/* FEW: gate/up, down (two launches); MANY: mx_gather before them (three). launch_count_out: how many were written. */
#define MX_PRODUCTS_LAUNCHES 3u
MUST_CHECK result_status mx_products_prepare(const struct mx_layer_description *description, uint64_t arena_byte_count,
					     const struct backend_operations *backend, struct device_card *card,
					     struct kernel_launch launches_out[MX_PRODUCTS_LAUNCHES],
					     uint32_t *launch_count_out);

/* router_select_b200 (arguments->router) and the rows' quantization as one launch */
MUST_CHECK result_status mx_route_quantize_prepare(const struct mx_route_quantize_arguments *arguments,
						   uint64_t arena_byte_count, const struct backend_operations *backend,
						   struct device_card *card, struct kernel_launch *launch_out);
MUST_CHECK result_status mx_quantize_prepare(const struct mx_quantize_arguments *arguments, uint64_t arena_byte_count,
					     const struct backend_operations *backend, struct device_card *card,
					     struct kernel_launch *launch_out);

/* Picks, grouping and the table of tiles of up to 128 rows of one expert: exl3_prefill_picks, exl3_prefill_group and
 * exl3_prefill_tiles on a record as router_wide_prepare takes it (every routed expert local, no always-on expert). */
#define ROUTER_TILES_LAUNCHES 3u
MUST_CHECK result_status router_tiles_prepare(const struct exl3_prefill_record *routing, uint64_t arena_byte_count,
					      const struct backend_operations *backend, struct device_card *card,
					      struct kernel_launch *launches_out);

#ifdef __cplusplus
}
static_assert(sizeof(struct mx_quantize_arguments) == 64 && sizeof(struct mx_route_quantize_arguments) == 152 &&
		      sizeof(struct mx_products_arguments) == 160 && sizeof(struct mx_gather_arguments) == 88,
	      "record ABI");
#else
_Static_assert(sizeof(struct mx_quantize_arguments) == 64 && sizeof(struct mx_route_quantize_arguments) == 152 &&
		       sizeof(struct mx_products_arguments) == 160 && sizeof(struct mx_gather_arguments) == 88,
	       "record ABI");
#endif
#endif
