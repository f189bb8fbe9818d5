/*
 * kernel_exl3_prefill.cu: the routed-expert layer for many rows (struct exl3_prefill_record): rows are grouped per
 * expert into tiles of 128 and every (one or two row tiles of an expert, 256 outputs of gate and up or 512 of down) is one
 * dense contraction on the fifth-generation tensor cores. The reference's counterpart is its tensor-core prefill family
 * (source/kernel_exl3_tcp.cuh), fixed to its model's shapes and to mma.sync; here a pair of CTAs
 *   - streams its rows' FP16 operands (pre-tiled in the tensor cores' no-swizzle K-major layout) into a ring of
 *     shared-memory stages, one bulk asynchronous copy a stage (one warp),
 *   - loads the trellis words of its outputs into registers a turn of the decode teams ahead, decodes them and stores
 *     them as the A operand blocks of the stage (sixteen warps in teams, a team a stage; the decode's fragment order
 *     makes every store a contiguous 128 bytes of the block),
 *   - multiplies with tcgen05.mma of cta_group::2 (one thread of the pair), FP32 accumulators in tensor memory, the stage
 *     released by tcgen05.commit,
 *   - reads the accumulators back with tcgen05.ld and applies the chain's FP32 epilogue (exl3_passes.cuh: Hadamard,
 *     scales, SwiGLU, down-side transform / route weight), four rows a warp, a row a warp to PREFILL_FEW_ROWS.
 * A single tile of at most eight rows takes none of it: mma.sync on what the decode leaves in registers (prefill_thin_products).
 * Arithmetic per value is the retained chain's; only the association of the FP32 sums over K is the tensor cores'.
 * Every wait is bounded: one that runs out raises exl3_wait_expired, the CTA stores nothing, waits (bounded) for what
 * it has in flight, frees its tensor memory and returns.
 */
#include "exl3_passes.cuh"
#include "router_device.cuh"

#define PREFILL_FIRST_DECODE_WARP 2u /* behind the copy warp and the issuing warp */
#define PREFILL_DECODE_WARPS 16u
#define PREFILL_DECODE_THREADS (PREFILL_DECODE_WARPS * EXL3_WARP)
#define PREFILL_GROUP_THREADS 256u

struct prefill_shared {
	uint64_t full[EXL3_PREFILL_MOST_STAGES]; /* the stage's weights are decoded and its rows have landed; rank 0: the other CTA's too */
	uint64_t free[EXL3_PREFILL_MOST_STAGES]; /* the products that read it are done */
	uint64_t done; /* every product of the pair is done */
	uint32_t tensor_memory;
	volatile uint32_t failed;
	uint32_t expired; /* an earlier wait had run out when the CTA began */
	uint32_t armed; /* stages whose row copies were started */
	uint32_t stages; /* of the ring */
	/* of the CTA's 128 outputs: gate's, up's and down's input-side scales; down: of its two groups */
	__half __align__(16) scales[3][EXL3_TRANSFORM];
};

/* The epilogue's scales, brought beside the K loop: read by the epilogue from memory they were its longest wait (1500 cycles
 * each time, four times in a row for a warp's rows). A decode warp a run of 256 bytes, half its lanes; complete at the
 * decode warps' barrier behind the K loop. */
__device__ __forceinline__ void prefill_fetch_scales(prefill_shared *shared, uint32_t place, const __half *scales)
{
	const uint32_t lane = threadIdx.x % EXL3_WARP;
	if (threadIdx.x / EXL3_WARP == PREFILL_FIRST_DECODE_WARP + place && lane < 16u)
		asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_address(shared->scales[place] + lane * 8u)),
			     "l"(scales + lane * 8u)
			     : "memory");
}

struct prefill_view {
	const struct exl3_prefill_parts parts;
	unsigned char *workspace;
	uint32_t experts; /* held here: routed + always-on */
	uint32_t pairs_per_row;
	uint32_t live;
	uint32_t widest; /* the larger intermediate width */
};

__device__ __forceinline__ prefill_view prefill_view_of(const struct exl3_prefill_record &record, unsigned char *arena)
{
	const struct step_block step = *reinterpret_cast<const struct step_block *>(arena + record.step_offset);
	const uint32_t widest = max(record.inner_size, record.shared_inner_size);
	prefill_view view = { exl3_prefill_parts_of(record.row_capacity, record.picks, record.shared_count,
						    record.local_count, record.input_size, widest),
			      arena + record.workspace_offset, record.local_count + record.shared_count,
			      record.picks + record.shared_count, min(step.row_count, record.row_capacity), widest };
	return view;
}

/* The first act of the launches that may each be given their places while the one before them still runs: all of that one
 * first; then the next may take its places. */
__device__ __forceinline__ void prefill_follow()
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

/* ------------------------------------------------------------------ routing */

extern "C" __global__ void __launch_bounds__(ROUTER_B200_THREADS)
	exl3_prefill_picks(struct exl3_prefill_record record, unsigned char *arena)
{
	__shared__ uint32_t chosen[ROUTER_B200_THREADS / WARP][ROUTER_B200_MAXIMUM_PICKS];
	__shared__ float weight[ROUTER_B200_THREADS / WARP][ROUTER_B200_MAXIMUM_PICKS];
	prefill_follow();
	const struct step_block step = *reinterpret_cast<const struct step_block *>(arena + record.step_offset);
	const uint32_t live = min(step.row_count, record.row_capacity);
	const uint32_t warp = threadIdx.x / WARP, lane = threadIdx.x % WARP;
	const uint32_t row = blockIdx.x * (blockDim.x / WARP) + warp;
	if (row >= live)
		return;
	router_row(reinterpret_cast<const float *>(arena + record.scores_offset) + (uint64_t)row * record.expert_count,
		   record.bias_offset != 0 ? reinterpret_cast<const float *>(arena + record.bias_offset) : nullptr,
		   record.expert_count, record.picks, record.scoring, record.route_scale, lane, chosen[warp], weight[warp],
		   reinterpret_cast<uint32_t *>(arena + record.picks_offset) + (uint64_t)row * record.picks,
		   reinterpret_cast<float *>(arena + record.weights_offset) + (uint64_t)row * record.picks);
}

/* A block an expert: its entries in ascending row order (a row holds an expert at most once) and their count. */
extern "C" __global__ void __launch_bounds__(PREFILL_GROUP_THREADS)
	exl3_prefill_group(struct exl3_prefill_record record, unsigned char *arena)
{
	__shared__ uint32_t warp_total[PREFILL_GROUP_THREADS / WARP];
	prefill_follow();
	const prefill_view view = prefill_view_of(record, arena);
	const uint32_t expert = blockIdx.x, lane = threadIdx.x % WARP, warp = threadIdx.x / WARP;
	const uint32_t *const picked = reinterpret_cast<const uint32_t *>(arena + record.picks_offset);
	const float *const weights = reinterpret_cast<const float *>(arena + record.weights_offset);
	struct exl3_prefill_entry *const entries =
		reinterpret_cast<struct exl3_prefill_entry *>(view.workspace + view.parts.entries) +
		(uint64_t)expert * record.row_capacity;
	uint32_t base = 0;
	for (uint32_t first = 0; first < view.live; first += PREFILL_GROUP_THREADS) {
		const uint32_t row = first + threadIdx.x;
		bool found = false;
		uint32_t slot = 0;
		float route_weight = 1.0f;
		if (row < view.live) {
			if (expert >= record.local_count) {
				found = true;
				slot = record.picks + (expert - record.local_count);
			} else {
				for (uint32_t place = 0; place < record.picks; place++)
					if (picked[(uint64_t)row * record.picks + place] == record.local_first + expert) {
						found = true;
						slot = place;
						route_weight = weights[(uint64_t)row * record.picks + place];
					}
			}
		}
		const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, found);
		if (lane == 0)
			warp_total[warp] = (uint32_t)__popc(ballot);
		__syncthreads();
		uint32_t before = 0, total = 0;
		for (uint32_t other = 0; other < PREFILL_GROUP_THREADS / WARP; other++) {
			before += other < warp ? warp_total[other] : 0u;
			total += warp_total[other];
		}
		if (found) {
			struct exl3_prefill_entry entry;
			entry.pair = row * view.pairs_per_row + slot;
			entry.route_weight = route_weight;
			entries[base + before + (uint32_t)__popc(ballot & ((1u << lane) - 1u))] = entry;
		}
		base += total;
		__syncthreads();
	}
	if (threadIdx.x == 0)
		reinterpret_cast<uint32_t *>(view.workspace + view.parts.counts)[expert] = base;
}

/* One block: the tile table in ascending expert order and the tile count. */
extern "C" __global__ void __launch_bounds__(ROUTER_B200_THREADS)
	exl3_prefill_tiles(struct exl3_prefill_record record, unsigned char *arena)
{
	__shared__ uint32_t warp_total[ROUTER_B200_THREADS / WARP];
	prefill_follow();
	const prefill_view view = prefill_view_of(record, arena);
	uint32_t *const counts = reinterpret_cast<uint32_t *>(view.workspace + view.parts.counts);
	struct exl3_prefill_tile *const tiles =
		reinterpret_cast<struct exl3_prefill_tile *>(view.workspace + view.parts.tiles);
	const uint32_t expert = threadIdx.x, lane = threadIdx.x % WARP, warp = threadIdx.x / WARP;
	const uint32_t rows = expert < view.experts ? counts[expert] : 0u;
	const uint32_t mine = (rows + EXL3_PREFILL_TILE_ROWS - 1u) / EXL3_PREFILL_TILE_ROWS;
	uint32_t inclusive = mine;
	for (uint32_t distance = 1; distance < WARP; distance <<= 1) {
		const uint32_t other = __shfl_up_sync(0xFFFFFFFFu, inclusive, distance);
		if (lane >= distance)
			inclusive += other;
	}
	if (lane == WARP - 1u)
		warp_total[warp] = inclusive;
	__syncthreads();
	uint32_t before = 0, total = 0;
	for (uint32_t other = 0; other < ROUTER_B200_THREADS / WARP; other++) {
		before += other < warp ? warp_total[other] : 0u;
		total += warp_total[other];
	}
	const uint32_t first_tile = before + inclusive - mine;
	for (uint32_t index = 0; index < mine; index++) {
		struct exl3_prefill_tile tile;
		tile.expert = expert;
		tile.first_entry = index * EXL3_PREFILL_TILE_ROWS;
		tile.row_count = min(rows - tile.first_entry, EXL3_PREFILL_TILE_ROWS);
		tile.reserved_zero = 0;
		if (first_tile + index < view.parts.tile_capacity)
			tiles[first_tile + index] = tile;
	}
	if (threadIdx.x == 0)
		counts[view.experts] = min(total, view.parts.tile_capacity);
}

/* the intermediate width of a local expert's matrices */
__device__ __forceinline__ uint32_t prefill_inner_of(const struct exl3_prefill_record &record, uint32_t expert)
{
	return expert < record.local_count ? record.inner_size : record.shared_inner_size;
}

/* A unit's rows: one row tile, or two of one expert (0: the second of two). An expert's row tiles are taken two at a time: the pair of an
 * even-numbered tile that has a successor also takes the successor's rows, so that every decoded weight is multiplied
 * with 256 rows; the pair of an odd-numbered tile returns. */
__device__ __forceinline__ uint32_t prefill_tiles_of_unit(const prefill_view &view, const struct exl3_prefill_tile &tile,
							  uint32_t tile_index, uint32_t tile_count)
{
	if ((tile.first_entry / EXL3_PREFILL_TILE_ROWS) % 2u != 0u)
		return 0;
	const struct exl3_prefill_tile *const tiles =
		reinterpret_cast<const struct exl3_prefill_tile *>(view.workspace + view.parts.tiles);
	return tile_index + 1u < tile_count && tiles[tile_index + 1u].expert == tile.expert ? 2u : 1u;
}

/* Where a tile's operands lie: what a CTA of the pair takes for one stage (gate and up 32 inputs, down 64) is ONE run of bytes,
 * [matrix][pieces of eight inputs][half rows][16 bytes], the stages one behind the other. The second CTA's runs are in the second
 * tile's region, or behind the first CTA's for a single tile. (With a fixed place for each of 128 rows a stage of fewer
 * rows was up to eight copies, and their issue, 1070 cycles a stage, was what bounded the products.) */
struct prefill_rows {
	uint32_t half; /* rows a CTA takes, whole sixteens */
	uint64_t second; /* from a single tile's first run to the second CTA's */
};

__device__ __forceinline__ prefill_rows prefill_rows_of(uint32_t count, uint32_t row_count, uint32_t matrices, uint32_t inputs)
{
	prefill_rows rows;
	/* a tile of two has a CTA for itself: all of its rows count as the first half */
	rows.half = count == 1u ? (row_count + 31u) / 32u * 16u : EXL3_PREFILL_TILE_ROWS;
	rows.second = (uint64_t)inputs * matrices * rows.half * 2u;
	return rows;
}

/* byte of (row, input) of matrix m inside the tile's region */
__device__ __forceinline__ uint64_t prefill_operand_byte(const prefill_rows &rows, uint32_t matrices, uint32_t m, uint32_t row,
							 uint32_t input)
{
	const uint32_t rank = row / rows.half, piece = input / 8u;
	const uint32_t pieces = 2u * EXL3_PREFILL_STAGE_STEPS(matrices); /* of a stage */
	return rank * rows.second + (uint64_t)((piece / pieces * matrices + m) * pieces + piece % pieces) * (rows.half * 16u) +
	       (row - rank * rows.half) * 16u + input % 8u * 2u;
}

/* Four rows a warp, eight lanes a row: what a lane holds of a block of 128 channels is four runs of four channels, at
 * 32 k + 4 (lane % 8) (hadamard128_rows' layout). */
#define PREFILL_WARP_ROWS 4u
/* A tile of at most this many rows is finished a row a warp (hadamard128_warp), whose chain is a third as long; the bits are
 * the same. gate/up and down together, us, 17 experts of as many rows each, H 4096, I 2048, a row a warp / four rows a
 * warp: 12 rows 165.7 / 169.7, 16 167.4 / 170.5, 32 171.7 / 174.6, 33 176.7 / 179.4, 40 178.3 / 177.7, 48 179.7 / 178.9,
 * 64 184.2 / 182.4, 128 204.7 / 202.3 (65 and 80 rows, where four rows a warp begin a second turn, 187.9 / 190.0 and 189.6 /
 * 190.5). */
#define PREFILL_FEW_ROWS 32u
__device__ __forceinline__ void prefill_scales(const __half *scales, uint32_t first_channel, uint2 out[4])
{
#pragma unroll
	for (uint32_t k = 0; k < 4; k++)
		out[k] = *reinterpret_cast<const uint2 *>(scales + first_channel + 32u * k);
}

/* grid (tile capacity, ceil(H / 128 / 4) x EXL3_PREFILL_OPERAND_PARTS) x 128: x . suh, Hadamard, FP16 operands of gate and
 * of up. A warp takes one 128-channel block of a quarter of the tile's rows, four rows at a time; four rows' stores to a
 * piece of the operand blocks are 64 adjacent bytes. Bound by instruction issue beside the operands' way to memory: 4096
 * rows of H 4096, 36864 pairs, 1.14 GB written, 238 us (321 with a row a warp, a launch half each of gate and up
 * and the rows through shared memory). Rows beyond the tile's count are not written: what the products make of them
 * stays in their own columns of the accumulators, which nobody reads. */
extern "C" __global__ void __launch_bounds__(EXL3_TRANSFORM_THREADS)
	exl3_prefill_operands(struct exl3_prefill_record record, unsigned char *arena)
{
	prefill_follow();
	const prefill_view view = prefill_view_of(record, arena);
	const uint32_t tile_index = blockIdx.x;
	const uint32_t tile_count = reinterpret_cast<const uint32_t *>(view.workspace + view.parts.counts)[view.experts];
	if (tile_index >= tile_count)
		return;
	const struct exl3_prefill_tile tile =
		reinterpret_cast<const struct exl3_prefill_tile *>(view.workspace + view.parts.tiles)[tile_index];
	const uint32_t lane = threadIdx.x % EXL3_WARP, warp = threadIdx.x / EXL3_WARP;
	const uint32_t part = blockIdx.y % EXL3_PREFILL_OPERAND_PARTS;
	const uint32_t block = blockIdx.y / EXL3_PREFILL_OPERAND_PARTS * EXL3_TRANSFORM_WARPS + warp;
	const uint32_t H = record.input_size;
	constexpr uint32_t part_rows = EXL3_PREFILL_TILE_ROWS / EXL3_PREFILL_OPERAND_PARTS;
	if (block >= H / EXL3_TRANSFORM || part * part_rows >= tile.row_count)
		return;
	const uint32_t channel = block * EXL3_TRANSFORM + lane % 8u * 4u;
	const uint32_t bits_x2 = exl3_bits_x2(reinterpret_cast<const uint32_t *>(arena + record.widths_offset)[tile.expert]);
	const uint64_t codes = exl3_code_bytes(H, prefill_inner_of(record, tile.expert), bits_x2);
	const uint64_t *const table = reinterpret_cast<const uint64_t *>(arena + record.expert_table_offset) + 3u * tile.expert;
	uint2 scales[EXL3_PROJECTIONS][4];
#pragma unroll
	for (uint32_t m = 0; m < EXL3_PROJECTIONS; m++)
		prefill_scales(reinterpret_cast<const __half *>(arena + table[m] + codes), channel, scales[m]);
	const struct exl3_prefill_entry *const entries =
		reinterpret_cast<const struct exl3_prefill_entry *>(view.workspace + view.parts.entries) +
		(uint64_t)tile.expert * record.row_capacity + tile.first_entry;
	const __nv_bfloat16 *const input = reinterpret_cast<const __nv_bfloat16 *>(arena + record.input_offset) + channel;
	const prefill_rows rows = prefill_rows_of(prefill_tiles_of_unit(view, tile, tile_index, tile_count), tile.row_count,
						  EXL3_PROJECTIONS, H);
	unsigned char *const region = view.workspace + view.parts.gate_up_operands + (uint64_t)tile_index * H * 512u;
	const uint32_t end = min((part + 1u) * part_rows, tile.row_count);
	for (uint32_t first = part * part_rows; first < end; first += PREFILL_WARP_ROWS) {
		const uint32_t row = first + lane / 8u;
		const uint64_t source = (uint64_t)(entries[min(row, end - 1u)].pair / view.pairs_per_row) * H;
		uint2 raw[4];
#pragma unroll
		for (uint32_t k = 0; k < 4; k++)
			raw[k] = *reinterpret_cast<const uint2 *>(input + source + 32u * k);
#pragma unroll
		for (uint32_t m = 0; m < EXL3_PROJECTIONS; m++) {
			float v[4][4];
#pragma unroll
			for (uint32_t k = 0; k < 4; k++) {
				float scale[4];
				half4_values(scales[m][k], scale);
				v[k][0] = __fmul_rn(__uint_as_float(raw[k].x << 16), scale[0]);
				v[k][1] = __fmul_rn(__uint_as_float(raw[k].x & 0xFFFF0000u), scale[1]);
				v[k][2] = __fmul_rn(__uint_as_float(raw[k].y << 16), scale[2]);
				v[k][3] = __fmul_rn(__uint_as_float(raw[k].y & 0xFFFF0000u), scale[3]);
			}
			hadamard128_rows(v, lane);
#pragma unroll
			for (uint32_t k = 0; k < 4; k++) {
#pragma unroll
				for (uint32_t j = 0; j < 4; j++)
					v[k][j] = __fmul_rn(v[k][j], EXL3_NORMALIZATION);
				if (row < end)
					store_half4(reinterpret_cast<__half *>(
							    region + prefill_operand_byte(rows, EXL3_PROJECTIONS, m, row, channel + 32u * k)),
						    v[k]);
			}
		}
	}
}

/* ------------------------------------------------------------------ tensor-core products */

/* A product unit belongs to a CTA PAIR (tcgen05 cta_group::2, one instruction over two SMs): the weights are the
 * instruction's M side, 256 outputs of which each CTA decodes its own 128, and the rows are its N side, up to two row
 * tiles of one expert (256 rows) of which each CTA brings its own half. So a decoded weight meets 256 rows, a row's
 * operands meet 256 outputs (gate/up; down: 512), and each SM's shared memory gives an instruction 64 bytes a cycle
 * (its 128 outputs and its 128 rows per 128 cycles). One CTA on its own with two row tiles of 128 x 128 products needs
 * 128 bytes a cycle for the instructions alone, all there is, and takes every row's operands from L2 twice as often.
 * The rows' number is the instruction's N, so a last tile of few rows costs the tensor cores little; the decode is the
 * same for any. 4096 rows of H 4096, I 2048, 256 experts of 8: gate/up 2202 us with single CTAs, 1812 so; down 1211,
 * 993. Neither end is full (1024 rows of 32 experts: 67 % of the issue slots, the tensor cores 43 % of the cycles): a
 * stage's turn in the ring, about 600 cycles for 64 inputs of which the products take 512 at most, and a unit's beginning,
 * epilogue and release lie between them: a third of a unit of 256 rows (gate/up 77 k cycles in its K loop and 41 k beside it,
 * down 41 and 27), a tenth of one of 9 to 32 (78 and 9, 42 and 9). */
#define PREFILL_PAIR 2u /* CTAs of a unit */
#define PREFILL_SUM_COLUMNS 256u /* tensor-memory columns of one accumulator: a row a column */

/* Shared-memory matrix descriptor of operands at a 16-byte aligned address, in two words, the second constant: no
 * swizzle, K-major, piece_bytes between the two 16-byte K pieces of a K = 16 step, 128 bytes between groups of eight rows
 * (or outputs). Places in the rings are constant numbers of 16-byte units apart. */
#define PREFILL_DESCRIPTOR_HIGH ((128u >> 4) | 1u << 14)
__device__ __forceinline__ uint32_t prefill_descriptor_low(const void *operands, uint32_t piece_bytes)
{
	return smem_address(operands) >> 4 | (piece_bytes >> 4) << 16;
}

/* FP16 A and B, both K-major, FP32 accumulators, M = 256, N = the pair's rows (a multiple of 32) */
__device__ __forceinline__ uint32_t prefill_instruction(uint32_t rows)
{
	return (1u << 4) | ((rows >> 3) << 17) | ((256u >> 4) << 24);
}

__device__ __forceinline__ void tensor_fence_before()
{
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tensor_fence_after()
{
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

/* accumulate 0: the sums begin with this product */
__device__ __forceinline__ void tensor_multiply(uint32_t sums, uint32_t a, uint32_t b, uint32_t instruction, uint32_t accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
		     "setp.ne.b32 p, %4, 0;\n\t"
		     "mov.b64 a, {%1, %5};\n\t"
		     "mov.b64 b, {%2, %5};\n\t"
		     "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n\t}" ::"r"(sums),
		     "r"(a), "r"(b), "r"(instruction), "r"(accumulate), "n"(PREFILL_DESCRIPTOR_HIGH)
		     : "memory");
}

/* arrives at this barrier of the CTAs of `ranks` (a bit each) once the products this thread issued so far are done */
__device__ __forceinline__ void tensor_commit(uint64_t *barrier, uint32_t ranks)
{
	asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
			     smem_address(barrier)),
		     "h"((uint16_t)ranks)
		     : "memory");
}

__device__ __forceinline__ void decode_sync()
{
	asm volatile("bar.sync 1, %0;" ::"n"(PREFILL_DECODE_THREADS) : "memory");
}

/* one lane of a converged warp, the same one every time */
__device__ __forceinline__ bool prefill_elected()
{
	uint32_t elected;
	asm volatile("{\n\t.reg .pred p;\n\t"
		     "elect.sync _|p, 0xFFFFFFFF;\n\t"
		     "selp.u32 %0, 1, 0, p;\n\t}"
		     : "=r"(elected));
	return elected != 0;
}

/* a whole warp's wait: its lanes go on, or give up, together */
template <bool ACROSS = false> __device__ __forceinline__ bool warp_wait(uint64_t *barrier, uint32_t parity)
{
	return __all_sync(0xFFFFFFFFu, barrier_wait<ACROSS>(barrier, parity)) != 0;
}

/* whether the phase, which arrivals of both CTAs complete, has completed by now, without a wait; pair_acquire follows */
__device__ __forceinline__ uint32_t pair_barrier_test(uint32_t barrier, uint32_t parity)
{
	uint32_t complete;
	asm volatile("{\n\t.reg .pred p;\n\t"
		     "mbarrier.test_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n\t"
		     "selp.u32 %0, 1, 0, p;\n\t}"
		     : "=r"(complete)
		     : "r"(barrier), "r"(parity)
		     : "memory");
	return complete;
}

/* a value every lane holds, as one the compiler knows to be the warp's (an operand of the tensor cores' instructions) */
__device__ __forceinline__ uint32_t warp_value(uint32_t value)
{
	return __shfl_sync(0xFFFFFFFFu, value, 0);
}

__device__ __forceinline__ void pair_sync()
{
	asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

/* the other CTA's (rank's) address of a variable of this one's */
__device__ __forceinline__ uint32_t pair_address(const volatile void *here, uint32_t rank)
{
	uint32_t there;
	asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
		     : "=r"(there)
		     : "r"((uint32_t)__cvta_generic_to_shared(const_cast<const void *>(here))), "r"(rank));
	return there;
}

/* pair_arrive arrives at a barrier of the other CTA's; what this thread has seen in its own CTA's shared memory is in
 * place for the thread that finds the phase complete there and then calls pair_acquire. Both fences order shared memory
 * alone. The arrival's own .release.cluster, or fence.acq_rel.cluster before it, waits for all of memory and holds the one
 * warp that arrives up for longer than a stage (4096 rows of 256 experts: 7.08 ms; that fence once for all the stages in
 * place, 5.52), the waits' own .acquire.cluster costs 1 % (4.96); so 4.93, and 4.92 with no ordering at all. */
__device__ __forceinline__ void pair_arrive(uint32_t there)
{
	asm volatile("fence.release.sync_restrict::shared::cta.cluster;\n\t"
		     "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(there)
		     : "memory");
}

__device__ __forceinline__ void pair_acquire()
{
	asm volatile("fence.acquire.sync_restrict::shared::cluster.cluster;" ::: "memory");
}

/* Dynamic shared memory of a product CTA: MATRICES x GROUPS = 2 accumulators, gate and up of 128 outputs or down of
 * 2 x 128; a ring of stages of 32 (gate and up) or 64 inputs (EXL3_PREFILL_STAGE_STEPS), each
 *   [matrix] the CTA's rows (up to 128 x 32 or 64 FP16, 8 or 16 KB): one bulk copy, mostly from L2
 *   [matrix x group] decoded weights, 128 outputs by as many inputs in the same layout: written by the decode warps
 * Rows and weights share the stage so that the issuing warp waits for ONE barrier a stage: a wait on a barrier that is
 * long complete takes it 150 cycles, three of them and the issue of four products 730, where the products of 256 rows
 * last 512. The trellis words do not pass here: the start of a bulk copy takes a warp 300 to 500 cycles, whatever the
 * bytes, and a stage's words were four runs (5 copies a stage: 650 cycles a stage; 12: 900). */
template <uint32_t MATRICES, uint32_t GROUPS> struct prefill_rings {
	static constexpr uint32_t steps = EXL3_PREFILL_STAGE_STEPS(MATRICES); /* of 16 inputs */
	static constexpr uint32_t block = steps * 4096u; /* of 128 rows or outputs */
	static constexpr uint32_t weights_at = MATRICES * block; /* in a stage, behind the rows */
	static constexpr uint32_t stage = weights_at + MATRICES * GROUPS * block;
	static constexpr uint32_t parts = MATRICES * GROUPS * steps; /* of a stage's weights, a decode warp each */
	static constexpr uint32_t teams = PREFILL_DECODE_WARPS / parts; /* of decode warps */
	static constexpr uint32_t stages = EXL3_PREFILL_DYNAMIC_BYTES / stage;
	static_assert(MATRICES * GROUPS * PREFILL_SUM_COLUMNS == 512u, "tensor memory has 512 columns");
	static_assert(stages <= EXL3_PREFILL_MOST_STAGES && MATRICES * GROUPS == 2u, "the rings' barriers; a stage's parts");
};

/* The K loop of one CTA of the pair. matrices[m]: the codes of matrix m (`outputs` outputs), of which this CTA decodes
 * the `groups` (0 .. GROUPS) groups of 128 outputs from group `first_group`; `sums`: GROUPS, or the groups either CTA
 * decodes if that is less; row_runs: this CTA's `half` rows (half the pair's, a multiple of 16) of the operands, a run a
 * stage; `blocks` stages. Warp 0 copies the rows' operands; warp 1 issues the products (rank 0) or
 * tells rank 0 which of this CTA's stages are in place (rank 1); warps 2 .. copy trellis words and decode. On return
 * the decode warps know whether the accumulators (PREFILL_SUM_COLUMNS apart from shared->tensor_memory; lane: output,
 * column: row of the pair) are complete; the other warps return false. All threads of both CTAs call. */
template <uint32_t BX2, uint32_t MATRICES, uint32_t GROUPS>
__device__ __forceinline__ bool prefill_products(const unsigned char *const (&matrices)[MATRICES], uint32_t outputs,
						 uint32_t first_group, uint32_t groups, uint32_t sums,
						 const unsigned char *row_runs, uint32_t half,
						 uint32_t blocks, uint32_t rank, unsigned char *dynamic_shared,
						 prefill_shared *shared)
{
	typedef exl3_ring<BX2> ring;
	typedef prefill_rings<MATRICES, GROUPS> rings;
	constexpr uint32_t S = rings::stages;
	const uint32_t lane = threadIdx.x % EXL3_WARP, warp = threadIdx.x / EXL3_WARP;
	const uint64_t step_words = (uint64_t)(outputs / EXL3_TILE) * ring::words; /* of one step of 16 inputs */
	const uint32_t accumulators = shared->tensor_memory;

	if (warp == 0) {
		/* the rows' operands: a copy a stage */
		if (lane == 0) {
			const uint32_t bytes = MATRICES * rings::steps * 32u * half;
			uint32_t block = 0;
			for (; block < blocks; block++) {
				const uint32_t stage = block % S;
				if (block >= S && !barrier_wait(&shared->free[stage], (block / S - 1u) & 1u))
					break;
				barrier_expect(&shared->full[stage], bytes);
				bulk_load(dynamic_shared + stage * rings::stage, row_runs + (uint64_t)block * bytes, bytes,
					  &shared->full[stage]);
			}
			shared->armed = block;
			if (block < blocks)
				shared->failed = 1;
		}
		return false;
	}
	if (warp == 1 && rank != 0) {
		/* rank 0 issues for both: a stage's arrival there says that this CTA's part of it is in place. This warp has seen
		 * the stage's phase complete, so the decode warps' stores (each behind its writer's proxy fence) and the rows'
		 * copy happened before its arrival, whose release at cluster scope and the acquire behind rank 0's wait carry that
		 * across. (The decode warps themselves have loads and stores in flight that a release would wait for.) */
		bool good = true;
		const uint32_t there = pair_address(shared->full, 0);
		for (uint32_t block = 0; block < blocks && good; block++) {
			good = warp_wait(&shared->full[block % S], (block / S) & 1u);
			if (good && lane == 0)
				pair_arrive(there + block % S * 8u);
			__syncwarp();
		}
		if (!good)
			shared->failed = 1;
		return false;
	}
	if (warp == 1) {
		/* This warp bounds the products where the rows are few. It has one issue slot in five or six beside the decode
		 * warps of its scheduler, so what counts is how many instructions a stage takes: counters instead of remainders,
		 * sums of descriptors made once, and the next stage's barrier asked for before this stage's products go out. */
		bool good = true;
		uint32_t ready = 0, stage = 0, parity = 0, accumulate = 0;
		const uint32_t instruction = warp_value(prefill_instruction(PREFILL_PAIR * half));
		const uint32_t r_low = warp_value(prefill_descriptor_low(dynamic_shared, half * 16u));
		const uint32_t w_low = warp_value(prefill_descriptor_low(dynamic_shared + rings::weights_at, 2048u));
		const uint32_t r_step = warp_value(2u * half), columns = warp_value(accumulators), live = warp_value(sums);
		const uint32_t full = warp_value(smem_address(shared->full)), r_second = MATRICES > 1u ? rings::steps * r_step : 0u;
		for (uint32_t left = blocks; left != 0; left--) {
			if (ready == 0) {
				good = warp_wait<true>(&shared->full[stage], parity);
				if (!good)
					break;
			}
			const uint32_t r = r_low + stage * (rings::stage >> 4), w = w_low + stage * (rings::stage >> 4);
			uint64_t *const freed = &shared->free[stage];
			stage++;
			if (stage == S)
				stage = 0, parity ^= 1u;
			pair_acquire();
			ready = pair_barrier_test(full + stage * 8u, parity);
			tensor_fence_after();
			if (prefill_elected()) {
#pragma unroll
				for (uint32_t step = 0; step < rings::steps; step++)
					tensor_multiply(columns, w + step * 256u, r + step * r_step, instruction, step == 0u ? accumulate : 1u);
				if (GROUPS == 1u || live > 1u)
#pragma unroll
					for (uint32_t step = 0; step < rings::steps; step++)
						tensor_multiply(columns + PREFILL_SUM_COLUMNS, w + (rings::steps + step) * 256u,
								r + r_second + step * r_step, instruction, step == 0u ? accumulate : 1u);
				tensor_commit(freed, 3u);
				if (left == 1u)
					tensor_commit(&shared->done, 3u);
			}
			accumulate = 1u;
			ready = __all_sync(0xFFFFFFFFu, left != 1u && ready != 0) ? 1u : 0u;
		}
		if (!good) {
			/* neither CTA stores anything; what was issued is waited for before either goes */
			if (lane == 0) {
				shared->failed = 1;
				asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(pair_address(&shared->failed, 1)), "r"(1u)
					     : "memory");
			}
			__syncwarp();
			if (prefill_elected())
				tensor_commit(&shared->done, 3u);
			__syncwarp();
		}
		(void)warp_wait(&shared->done, 0u);
		return false;
	}

	/* decode: the sixteen warps are teams of a warp a part, four for gate and up and two for down; team q of T decodes the
	 * WHOLE stages q, q + T, ..., so that the teams work on different stages at once and a warp crosses a barrier and a
	 * proxy fence once per stage of eight tiles. A warp's part of a stage is the eight adjacent tiles of one (matrix, group, step).
	 * A lane loads its ring words straight into registers, a tile's words for the team's next stage as soon as this one's are
	 * decoded: 128 inputs, more than a microsecond, ahead. */
	{
		static_assert(PREFILL_DECODE_WARPS == rings::parts * rings::teams, "a part a warp");
		const uint32_t decoder = warp - PREFILL_FIRST_DECODE_WARP, team = decoder / rings::parts, member = decoder % rings::parts;
		const uint32_t step = member % rings::steps, g = GROUPS > 1u ? member / rings::steps : 0u;
		const uint32_t m = MATRICES > 1u ? member / rings::steps : 0u;
		const uint32_t begin = ring::begin(lane);
		const uint32_t word_index = begin / 32u, shift = begin % 32u, next_index = (word_index + 1u) % ring::words;
		const bool taken = g < groups; /* the CTA has this group */
		unsigned char *const to_part = dynamic_shared + rings::weights_at + (m + g) * rings::block + step * 4096u + lane * 4u;
		const uint32_t *words_at =
			reinterpret_cast<const uint32_t *>(MATRICES > 1u && m != 0u ? matrices[MATRICES - 1u] : matrices[0]) +
			(uint64_t)(team * rings::steps + step) * step_words +
			(uint64_t)(first_group + g) * EXL3_GROUP_TILES * ring::words;
		const uint64_t turn_words = (uint64_t)(rings::teams * rings::steps) * step_words;
		bool good = true;
		uint32_t words[EXL3_GROUP_TILES][2];
		if (taken && team < blocks)
#pragma unroll
			for (uint32_t tile = 0; tile < EXL3_GROUP_TILES; tile++) {
				words[tile][0] = __ldg(words_at + tile * ring::words + word_index);
				words[tile][1] = __ldg(words_at + tile * ring::words + next_index);
			}
		for (uint32_t block = team; block < blocks; block += rings::teams) {
			const uint32_t stage = block % S;
			if (block + rings::teams < blocks)
				words_at += turn_words; /* of the next turn; the last loads its own once more */
			if (block >= S) {
				good = warp_wait(&shared->free[stage], (block / S - 1u) & 1u);
				if (!good)
					break;
			}
			unsigned char *const to_stage = to_part + stage * rings::stage;
#pragma unroll
			for (uint32_t tile = 0; tile < EXL3_GROUP_TILES; tile++) {
				if (!taken)
					continue;
				uint32_t fragment[4];
				exl3_decode_fragment<BX2>(words[tile][0], words[tile][1], shift, fragment);
				words[tile][0] = __ldg(words_at + tile * ring::words + word_index);
				words[tile][1] = __ldg(words_at + tile * ring::words + next_index);
				/* fragment f: outputs 16 tile + g + 8 (f % 2), inputs 16 step + 2 t + 8 (f / 2): the warp's 32
				 * words are the 128 bytes of one K piece of one group of eight outputs */
				uint32_t *const to = reinterpret_cast<uint32_t *>(to_stage + tile * 2u * 128u);
				to[0] = fragment[0];
				to[128u / 4u] = fragment[1];
				to[2048u / 4u] = fragment[2];
				to[(2048u + 128u) / 4u] = fragment[3];
			}
			asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
			__syncwarp();
			if (lane == 0)
				barrier_arrive(&shared->full[stage]);
		}
		if (good)
			good = barrier_wait(&shared->done, 0u);
		if (!good)
			shared->failed = 1;
		tensor_fence_after();
		asm volatile("cp.async.wait_all;" ::: "memory");
		decode_sync(); /* every decode warp has its verdict in, and the scales are in place */
		return shared->failed == 0;
	}
}

/* Begins a product CTA: barriers, tensor memory, and the pair's agreement on whether to run. All threads of both CTAs
 * call; false: an earlier wait ran out, the pair is to go (the flag is never cleared while the kernel file stays loaded:
 * later CTAs do not queue up behind the same fault, the host reads the flag and rejects the result). */
__device__ __forceinline__ bool prefill_begin(prefill_shared *shared, uint32_t rank, uint32_t stages, uint32_t parts)
{
	const uint32_t warp = threadIdx.x / EXL3_WARP;
	if (threadIdx.x == 0) {
		for (uint32_t stage = 0; stage < stages; stage++) {
			/* the warps of the team that decodes the stage, the rows' copies, at rank 0 the other CTA */
			barrier_init(&shared->full[stage], parts + (rank == 0 ? 2u : 1u));
			barrier_init(&shared->free[stage], 1);
		}
		barrier_init(&shared->done, 1);
		shared->failed = 0;
		shared->armed = 0;
		shared->stages = stages;
		shared->expired = *reinterpret_cast<volatile unsigned int *>(&exl3_wait_expired);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 1) {
		asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
				     smem_address(&shared->tensor_memory))
			     : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
	}
	tensor_fence_before();
	__syncthreads();
	pair_sync();
	tensor_fence_after();
	uint32_t other;
	asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(other) : "r"(pair_address(&shared->expired, rank ^ 1u)) : "memory");
	return (shared->expired | other) == 0;
}

/* `sums` accumulators of one row tile (first columns first_column, + PREFILL_SUM_COLUMNS, ...) into shared memory, FP32
 * [accumulator][row][EXL3_PREFILL_STAGING_ROW outputs]. A warp reads the 32 outputs of its quarter (warp % 4) and 32 of
 * the `rows` rows. Decode warps only; ends with their barrier. */
__device__ __forceinline__ void prefill_stage_out(uint32_t accumulators, uint32_t sums, uint32_t first_column, uint32_t rows,
						  float *staging)
{
	const uint32_t lane = threadIdx.x % EXL3_WARP, warp = threadIdx.x / EXL3_WARP;
	const uint32_t quarter = warp % 4u, column = (warp - PREFILL_FIRST_DECODE_WARP) / 4u * 32u;
	__syncwarp();
	if (column < rows)
		for (uint32_t m = 0; m < sums; m++) {
			uint32_t r[32];
			asm volatile(
				"tcgen05.ld.sync.aligned.32x32b.x32.b32 "
				"{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
				"%26,%27,%28,%29,%30,%31}, [%32];"
				: "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
				  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
				  "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
				  "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
				  "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
				: "r"(accumulators + ((quarter * 32u) << 16) + first_column + m * PREFILL_SUM_COLUMNS + column)
				: "memory");
			asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
			/* a lane an output: the 32 lanes of a row's store are 32 adjacent floats */
			float *const to = staging + (m * EXL3_PREFILL_TILE_ROWS + column) * EXL3_PREFILL_STAGING_ROW + quarter * 32u + lane;
#pragma unroll
			for (uint32_t index = 0; index < 32; index++)
				to[index * EXL3_PREFILL_STAGING_ROW] = __uint_as_float(r[index]);
		}
	tensor_fence_before();
	decode_sync();
}

/* All threads of both CTAs, at the end: wait (bounded) for what a failed CTA still has in flight, and for the other CTA,
 * whose products read this one's shared memory, then free the tensor memory. */
__device__ __forceinline__ void prefill_release(prefill_shared *shared)
{
	tensor_fence_before();
	__syncthreads();
	if (shared->failed != 0 && threadIdx.x == 0) {
		/* a stage whose other arrivals are missing holds this thread up to the bound, long past its copies' end */
		for (uint32_t back = 0; back < shared->stages && back < shared->armed; back++) {
			const uint32_t block = shared->armed - 1u - back;
			(void)barrier_wait(&shared->full[block % shared->stages], (block / shared->stages) & 1u);
		}
	}
	__syncthreads();
	pair_sync();
	if (threadIdx.x / EXL3_WARP == 1u) {
		tensor_fence_after();
		__syncwarp();
		asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(shared->tensor_memory) : "memory");
	}
}

struct prefill_tile_view {
	struct exl3_prefill_tile tile;
	const struct exl3_prefill_entry *entries; /* of the tile's rows */
	uint64_t gate, up, down; /* matrix offsets */
};

__device__ __forceinline__ prefill_tile_view prefill_tile_of(const struct exl3_prefill_record &record,
							     const unsigned char *arena, const prefill_view &view,
							     uint32_t tile_index)
{
	prefill_tile_view out;
	out.tile = reinterpret_cast<const struct exl3_prefill_tile *>(view.workspace + view.parts.tiles)[tile_index];
	out.entries = reinterpret_cast<const struct exl3_prefill_entry *>(view.workspace + view.parts.entries) +
		      (uint64_t)out.tile.expert * record.row_capacity + out.tile.first_entry;
	const uint64_t *const table = reinterpret_cast<const uint64_t *>(arena + record.expert_table_offset);
	out.gate = table[3u * out.tile.expert];
	out.up = table[3u * out.tile.expert + 1u];
	out.down = table[3u * out.tile.expert + 2u];
	return out;
}

/* The gate/up epilogue of one row tile and one group of 128 outputs, from the staged accumulators (gate rows, then up
 * rows): Hadamard, scales, SwiGLU, down-side transform, FP16 down operand blocks. Decode warps; four rows a warp, a row a warp to PREFILL_FEW_ROWS. */
__device__ __forceinline__ void prefill_gate_up_rows(const struct exl3_prefill_record &record, const prefill_view &view,
						     const prefill_shared *shared, const prefill_tile_view &tile,
						     uint32_t tile_index, uint32_t count, uint32_t group, float *staging)
{
	const uint32_t I = prefill_inner_of(record, tile.tile.expert);
	const uint32_t lane = threadIdx.x % EXL3_WARP, warp = threadIdx.x / EXL3_WARP;
	const uint32_t channel = group * EXL3_TRANSFORM + lane % 8u * 4u;
	const __half *const scales = shared->scales[0] + lane % 8u * 4u;
	const prefill_rows rows = prefill_rows_of(count, tile.tile.row_count, 1u, I);
	unsigned char *const region = view.workspace + view.parts.down_operands + (uint64_t)tile_index * view.widest * 256u;
	if (tile.tile.row_count <= PREFILL_FEW_ROWS) {
		const uint32_t at = lane * 4u;
		for (uint32_t row = warp - PREFILL_FIRST_DECODE_WARP; row < tile.tile.row_count; row += PREFILL_DECODE_WARPS) {
			const float4 g = *reinterpret_cast<const float4 *>(staging + row * EXL3_PREFILL_STAGING_ROW + at);
			const float4 u = *reinterpret_cast<const float4 *>(staging +
									   (EXL3_PREFILL_TILE_ROWS + row) * EXL3_PREFILL_STAGING_ROW + at);
			float gate[4] = { g.x, g.y, g.z, g.w }, up[4] = { u.x, u.y, u.z, u.w };
			float gate_scale[4], up_scale[4], down_scale[4], fed[4];
			load_half4(shared->scales[0] + at, gate_scale);
			load_half4(shared->scales[1] + at, up_scale);
			load_half4(shared->scales[2] + at, down_scale);
			hadamard128_warp(gate, lane);
			hadamard128_warp(up, lane);
			exl3_swiglu4(gate, up, gate_scale, up_scale, record.activation_limit, fed);
#pragma unroll
			for (uint32_t i = 0; i < 4; i++)
				fed[i] = __fmul_rn(fed[i], down_scale[i]);
			hadamard128_warp(fed, lane);
#pragma unroll
			for (uint32_t i = 0; i < 4; i++)
				fed[i] = __fmul_rn(fed[i], EXL3_NORMALIZATION);
			store_half4(reinterpret_cast<__half *>(
					    region + prefill_operand_byte(rows, 1u, 0u, row, group * EXL3_TRANSFORM + at)),
				    fed);
		}
		return;
	}
#pragma unroll 1
	for (uint32_t first = (warp - PREFILL_FIRST_DECODE_WARP) * PREFILL_WARP_ROWS; first < tile.tile.row_count;
	     first += PREFILL_DECODE_WARPS * PREFILL_WARP_ROWS) {
		const uint32_t row = first + lane / 8u; /* beyond the tile's count: a row of whatever stands there, not stored */
		/* the staged rows: up's, then gate's, which become the hidden values' */
		float *const gate_at = staging + row * EXL3_PREFILL_STAGING_ROW + lane % 8u * 4u;
		float *const up_at = gate_at + EXL3_PREFILL_TILE_ROWS * EXL3_PREFILL_STAGING_ROW;
		/* One copy of the transform for up, gate and the down-side one, and of the hidden step for four values: what these
		 * cost a unit of few rows is the fetch of their instructions (16 values of each unrolled: 10 to 13 k cycles an
		 * epilogue of up to 16 rows, 4 k so). What a lane stores here it alone reads again. */
#pragma unroll 1
		for (uint32_t pass = 0; pass < 3u; pass++) {
			float *const at = pass == 0u ? up_at : gate_at;
			if (pass == 2u)
#pragma unroll 1
				for (uint32_t k = 0; k < 4; k++) {
					float gate_scale[4], up_scale[4], down_scale[4], hidden[4];
					load_half4(scales + 32u * k, gate_scale);
					load_half4(scales + EXL3_TRANSFORM + 32u * k, up_scale);
					load_half4(scales + 2u * EXL3_TRANSFORM + 32u * k, down_scale);
					float4 *const to = reinterpret_cast<float4 *>(gate_at + 32u * k);
					const float4 g = *to, u = *reinterpret_cast<const float4 *>(up_at + 32u * k);
					float gate[4] = { g.x, g.y, g.z, g.w }, up[4] = { u.x, u.y, u.z, u.w };
					exl3_swiglu4(gate, up, gate_scale, up_scale, record.activation_limit, hidden);
					*to = make_float4(__fmul_rn(hidden[0], down_scale[0]), __fmul_rn(hidden[1], down_scale[1]),
							  __fmul_rn(hidden[2], down_scale[2]), __fmul_rn(hidden[3], down_scale[3]));
				}
			float v[4][4];
#pragma unroll
			for (uint32_t k = 0; k < 4; k++) {
				const float4 raw = *reinterpret_cast<const float4 *>(at + 32u * k);
				v[k][0] = raw.x, v[k][1] = raw.y, v[k][2] = raw.z, v[k][3] = raw.w;
			}
			hadamard128_rows(v, lane);
#pragma unroll
			for (uint32_t k = 0; k < 4; k++) {
				if (pass != 2u) {
					*reinterpret_cast<float4 *>(at + 32u * k) = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
				} else if (row < tile.tile.row_count) {
#pragma unroll
					for (uint32_t j = 0; j < 4; j++)
						v[k][j] = __fmul_rn(v[k][j], EXL3_NORMALIZATION);
					store_half4(reinterpret_cast<__half *>(region + prefill_operand_byte(rows, 1u, 0u, row, channel + 32u * k)),
						    v[k]);
				}
			}
		}
	}
}

/* The products of a single tile of at most PREFILL_THIN_ROWS rows, by mma.sync on what the decode leaves in registers: no
 * stage, no hand-over to another warp, no tensor memory. Sixteen warps, 16 outputs each of the two (matrix, group)s; a lane
 * holds its ring words and the rows' operands (two runs of 128 bytes a step, shared by eight warps in the L1) a turn of eight
 * steps ahead, and asks the L2 for the turn after the next, a lane a step. The sums go into the staged rows the epilogues read.
 * Decode warps only; ends with their barrier.
 * A warp walks ALL of K in one accumulator: the sums are then the same bits as the tensor cores' accumulators in tensor memory
 * (both instructions add sixteen products to an FP32 sum, with the same roundings; nothing documents it, the tests hold it at
 * every width), so a row's result does not depend on how many rows its expert has in the call. K shared out over eight warps,
 * a step's eight tiles a warp, is faster (below) but gives a row other bits in a short tile than in a long one.
 * Such a tile's time is its decode and what a unit costs beside it (a pair's beginning, 5 k cycles, the stages' hand-overs, a
 * fifth of its 70 k). 413 rows of 256 experts, 59 of 97 with at most eight rows: gate/up and down 538 and 311 us through the
 * stages, 519 and 298 so, 506 and 294 with K shared out; 4096 rows, 95 of 173: 1872 and 1002, 1843 and 991, 1824 and 977 (all
 * with stages of 64 inputs).
 * Without the L2's request 523 and 305. More than eight rows would be a second product a fragment. */
#define PREFILL_THIN_ROWS 8u
#define PREFILL_THIN_HALF 16u /* rows of the first CTA's half of such a tile's operands (prefill_rows_of) */
#define PREFILL_THIN_TURN 8u /* steps a lane holds: four take 603 and 339 us; K is a multiple of 128 inputs */
template <uint32_t BX2, uint32_t MATRICES, uint32_t GROUPS>
__device__ __forceinline__ void prefill_thin_products(const unsigned char *const (&matrices)[MATRICES], uint32_t outputs,
						      uint32_t first_group, uint32_t groups, const unsigned char *row_runs,
						      uint32_t row_count, uint32_t steps, unsigned char *dynamic_shared)
{
	typedef exl3_ring<BX2> ring;
	constexpr uint32_t stage_steps = EXL3_PREFILL_STAGE_STEPS(MATRICES);
	static_assert(PREFILL_DECODE_WARPS == MATRICES * GROUPS * EXL3_GROUP_TILES, "16 outputs a warp");
	static_assert(PREFILL_THIN_TURN % stage_steps == 0u && EXL3_TRANSFORM / EXL3_TILE % PREFILL_THIN_TURN == 0u,
		      "a turn is whole stages, K whole turns");
	const uint32_t lane = threadIdx.x % EXL3_WARP, decoder = threadIdx.x / EXL3_WARP - PREFILL_FIRST_DECODE_WARP;
	const uint32_t which = decoder / EXL3_GROUP_TILES, tile = decoder % EXL3_GROUP_TILES;
	const uint32_t g = GROUPS > 1u ? which : 0u, m = MATRICES > 1u ? which : 0u;
	if (g < groups) {
		const uint64_t step_words = (uint64_t)(outputs / EXL3_TILE) * ring::words;
		const uint32_t begin = ring::begin(lane);
		const uint32_t word_index = begin / 32u, shift = begin % 32u, next_index = (word_index + 1u) % ring::words;
		const uint64_t first = (uint64_t)(MATRICES > 1u && m != 0u ? matrices[MATRICES - 1u] : matrices[0]) +
				       ((uint64_t)(first_group + g) * EXL3_GROUP_TILES + tile) * ring::words * 4u;
		/* the warp's address, known to be one: a step's is one addition */
		const uint32_t *words = reinterpret_cast<const uint32_t *>((uint64_t)warp_value((uint32_t)(first >> 32)) << 32 |
									   warp_value((uint32_t)first));
		const uint32_t *ahead = words + (2u * PREFILL_THIN_TURN + lane % PREFILL_THIN_TURN) * step_words;
		/* step s stands in stage s / stage_steps: [matrix][pieces][half rows][16 bytes]; the lane's two words of it */
		constexpr uint32_t piece = PREFILL_THIN_HALF * 16u, stage_bytes = MATRICES * stage_steps * 2u * piece;
		const unsigned char *fed = row_runs + m * stage_steps * 2u * piece + lane / 4u * 16u + lane % 4u * 4u;
		float sums[4] = { 0.0f, 0.0f, 0.0f, 0.0f };
		uint32_t held[PREFILL_THIN_TURN][2], held_fed[PREFILL_THIN_TURN][2];
#pragma unroll
		for (uint32_t step = 0; step < PREFILL_THIN_TURN; step++) {
			const unsigned char *const at = fed + step / stage_steps * stage_bytes + step % stage_steps * 2u * piece;
			held[step][0] = __ldg(words + word_index);
			held[step][1] = __ldg(words + next_index);
			held_fed[step][0] = *reinterpret_cast<const uint32_t *>(at);
			held_fed[step][1] = *reinterpret_cast<const uint32_t *>(at + piece);
			words += step_words;
		}
#pragma unroll 1
		for (uint32_t left = steps / PREFILL_THIN_TURN; left != 0; left--) {
			if (left == 1u) /* the last turn loads its own once more */
				words -= PREFILL_THIN_TURN * step_words;
			else
				fed += PREFILL_THIN_TURN / stage_steps * stage_bytes;
			if (left > 2u && lane < PREFILL_THIN_TURN) {
				asm volatile("prefetch.global.L2 [%0];" ::"l"(ahead));
				ahead += PREFILL_THIN_TURN * step_words;
			}
#pragma unroll
			for (uint32_t step = 0; step < PREFILL_THIN_TURN; step++) {
				const unsigned char *const at = fed + step / stage_steps * stage_bytes + step % stage_steps * 2u * piece;
				uint32_t fragment[4];
				exl3_decode_fragment<BX2>(held[step][0], held[step][1], shift, fragment);
				held[step][0] = __ldg(words + word_index);
				held[step][1] = __ldg(words + next_index);
				words += step_words;
				mma_f16(sums, fragment, held_fed[step][0], held_fed[step][1]);
				held_fed[step][0] = *reinterpret_cast<const uint32_t *>(at);
				held_fed[step][1] = *reinterpret_cast<const uint32_t *>(at + piece);
			}
		}
#pragma unroll
		for (uint32_t c = 0; c < 4; c++) {
			const uint32_t row = lane % 4u * 2u + (c & 1u);
			if (row < row_count)
				reinterpret_cast<float *>(dynamic_shared)[(which * EXL3_PREFILL_TILE_ROWS + row) * EXL3_PREFILL_STAGING_ROW +
									  tile * EXL3_TILE + lane / 4u + (c >> 1) * 8u] = sums[c];
		}
	}
	asm volatile("cp.async.wait_all;" ::: "memory"); /* the scales */
	decode_sync();
}

/* gate and up of a unit's `count` row tiles (tile_index, + 1) by 256 outputs: this CTA's group is `group` */
template <uint32_t BX2>
__device__ __forceinline__ void prefill_gate_up(const struct exl3_prefill_record &record, unsigned char *arena,
						const prefill_view &view, uint32_t tile_index, uint32_t count, uint32_t group,
						uint32_t rank, unsigned char *dynamic_shared, prefill_shared *shared)
{
	const prefill_tile_view first = prefill_tile_of(record, arena, view, tile_index);
	const uint32_t H = record.input_size, I = prefill_inner_of(record, first.tile.expert);
	const uint32_t mine = group < I / EXL3_TRANSFORM ? 1u : 0u;
	const unsigned char *const matrices[2] = { arena + first.gate, arena + first.up };
	const prefill_rows rows = prefill_rows_of(count, first.tile.row_count, 2u, H);
	const unsigned char *const row_runs = view.workspace + view.parts.gate_up_operands +
					      (uint64_t)(tile_index + (count == 2u ? rank : 0u)) * H * 512u +
					      (count == 2u ? 0u : rank * rows.second);
	if (mine != 0) {
		const uint64_t codes = exl3_code_bytes(H, I, BX2), first_scale = group * EXL3_TRANSFORM;
		prefill_fetch_scales(shared, 0u, reinterpret_cast<const __half *>(arena + first.gate + codes) + H + first_scale);
		prefill_fetch_scales(shared, 1u, reinterpret_cast<const __half *>(arena + first.up + codes) + H + first_scale);
		prefill_fetch_scales(shared, 2u, reinterpret_cast<const __half *>(arena + first.down + exl3_code_bytes(I, H, BX2)) +
							 first_scale);
	}
	const bool complete = prefill_products<BX2, 2, 1>(matrices, I, group, mine, 1, row_runs, rows.half,
							  H / (prefill_rings<2, 1>::steps * EXL3_TILE), rank, dynamic_shared, shared);
	if (threadIdx.x / EXL3_WARP >= PREFILL_FIRST_DECODE_WARP && complete && mine != 0) {
		float *const staging = reinterpret_cast<float *>(dynamic_shared);
		for (uint32_t tile = 0; tile < count; tile++) {
			const prefill_tile_view rows_of = prefill_tile_of(record, arena, view, tile_index + tile);
			prefill_stage_out(shared->tensor_memory, 2, tile * EXL3_PREFILL_TILE_ROWS, rows_of.tile.row_count, staging);
			prefill_gate_up_rows(record, view, shared, rows_of, tile_index + tile, count, group, staging);
			decode_sync(); /* the staging rows are read: the next tile may overwrite them */
		}
	}
	prefill_release(shared);
}

/* The down epilogue of one row tile from the staged accumulators, a group each: output transform, scale, route weight, FP32
 * pair outputs. Decode warps. */
__device__ __forceinline__ void prefill_down_rows(const prefill_shared *shared, const prefill_tile_view &rows_of,
						  uint32_t first_group, uint32_t groups, uint32_t H, float *outputs,
						  const float *staging)
{
	const uint32_t lane = threadIdx.x % EXL3_WARP, warp = threadIdx.x / EXL3_WARP;
	for (uint32_t g = 0; g < groups; g++) {
		const uint32_t channel = (first_group + g) * EXL3_TRANSFORM + lane % 8u * 4u;
		const __half *const scales = shared->scales[g] + lane % 8u * 4u;
		if (rows_of.tile.row_count <= PREFILL_FEW_ROWS) {
			float scale[4];
			load_half4(shared->scales[g] + lane * 4u, scale);
			for (uint32_t row = warp - PREFILL_FIRST_DECODE_WARP; row < rows_of.tile.row_count;
			     row += PREFILL_DECODE_WARPS) {
				const struct exl3_prefill_entry entry = rows_of.entries[row];
				const float4 raw = *reinterpret_cast<const float4 *>(
					staging + (g * EXL3_PREFILL_TILE_ROWS + row) * EXL3_PREFILL_STAGING_ROW + lane * 4u);
				float v[4] = { raw.x, raw.y, raw.z, raw.w };
				hadamard128_warp(v, lane);
#pragma unroll
				for (uint32_t i = 0; i < 4; i++)
					v[i] = __fmul_rn(__fmul_rn(__fmul_rn(v[i], EXL3_NORMALIZATION), scale[i]),
							 entry.route_weight);
				*reinterpret_cast<float4 *>(outputs + (uint64_t)entry.pair * H +
							    (first_group + g) * EXL3_TRANSFORM + lane * 4u) =
					make_float4(v[0], v[1], v[2], v[3]);
			}
			continue;
		}
		for (uint32_t from = (warp - PREFILL_FIRST_DECODE_WARP) * PREFILL_WARP_ROWS; from < rows_of.tile.row_count;
		     from += PREFILL_DECODE_WARPS * PREFILL_WARP_ROWS) {
			const uint32_t row = from + lane / 8u;
			const struct exl3_prefill_entry entry = rows_of.entries[min(row, rows_of.tile.row_count - 1u)];
			const float *const at =
				staging + (g * EXL3_PREFILL_TILE_ROWS + row) * EXL3_PREFILL_STAGING_ROW + lane % 8u * 4u;
			float v[4][4];
#pragma unroll
			for (uint32_t k = 0; k < 4; k++) {
				const float4 raw = *reinterpret_cast<const float4 *>(at + 32u * k);
				v[k][0] = raw.x, v[k][1] = raw.y, v[k][2] = raw.z, v[k][3] = raw.w;
			}
			hadamard128_rows(v, lane);
#pragma unroll
			for (uint32_t k = 0; k < 4; k++) {
				float scale[4];
				load_half4(scales + 32u * k, scale);
#pragma unroll
				for (uint32_t j = 0; j < 4; j++)
					v[k][j] = __fmul_rn(__fmul_rn(__fmul_rn(v[k][j], EXL3_NORMALIZATION), scale[j]),
							    entry.route_weight);
				if (row < rows_of.tile.row_count)
					*reinterpret_cast<float4 *>(outputs + (uint64_t)entry.pair * H + channel + 32u * k) =
						make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
			}
		}
	}
}

/* down of a unit's `count` row tiles by 512 outputs: this CTA's groups are first_group, + 1; `sums`: 2, or 1 where the
 * last unit has no second group for either CTA */
template <uint32_t BX2>
__device__ __forceinline__ void prefill_down(const struct exl3_prefill_record &record, unsigned char *arena,
					     const prefill_view &view, uint32_t tile_index, uint32_t count,
					     uint32_t first_group, uint32_t sums, uint32_t rank,
					     unsigned char *dynamic_shared, prefill_shared *shared)
{
	const prefill_tile_view first = prefill_tile_of(record, arena, view, tile_index);
	const uint32_t H = record.input_size, I = prefill_inner_of(record, first.tile.expert);
	const uint32_t groups = first_group < H / EXL3_TRANSFORM ? min(2u, H / EXL3_TRANSFORM - first_group) : 0u;
	const uint32_t warp = threadIdx.x / EXL3_WARP;
	const unsigned char *const matrices[1] = { arena + first.down };
	const prefill_rows rows = prefill_rows_of(count, first.tile.row_count, 1u, I);
	const unsigned char *const row_runs = view.workspace + view.parts.down_operands +
					      (uint64_t)(tile_index + (count == 2u ? rank : 0u)) * view.widest * 256u +
					      (count == 2u ? 0u : rank * rows.second);
	for (uint32_t g = 0; g < groups; g++)
		prefill_fetch_scales(shared, g, reinterpret_cast<const __half *>(arena + first.down + exl3_code_bytes(I, H, BX2)) + I +
							 (first_group + g) * EXL3_TRANSFORM);
	const bool complete = prefill_products<BX2, 1, 2>(matrices, H, first_group, groups, sums, row_runs, rows.half,
							  I / (prefill_rings<1, 2>::steps * EXL3_TILE), rank, dynamic_shared, shared);
	if (warp >= PREFILL_FIRST_DECODE_WARP && complete) {
		float *const staging = reinterpret_cast<float *>(dynamic_shared);
		float *const outputs = reinterpret_cast<float *>(arena + record.pair_output_offset);
		for (uint32_t tile = 0; tile < count && groups != 0; tile++) {
			const prefill_tile_view rows_of = prefill_tile_of(record, arena, view, tile_index + tile);
			prefill_stage_out(shared->tensor_memory, groups, tile * EXL3_PREFILL_TILE_ROWS, rows_of.tile.row_count,
					  staging);
			prefill_down_rows(shared, rows_of, first_group, groups, H, outputs, staging);
			decode_sync();
		}
	}
	prefill_release(shared);
}

/* gate and up of a tile of few rows (its own only one) by the 128 outputs of group `group`. Decode warps. The tiles of few rows
 * and the others part at their launch's beginning: with both forms behind one switch over the widths gate/up's launch spilled
 * 48 bytes of registers (32 experts of 1024 rows: gate/up 427 us, 422 so). */
template <uint32_t BX2>
__device__ __forceinline__ void prefill_thin_gate_up(const struct exl3_prefill_record &record, unsigned char *arena,
						     const prefill_view &view, uint32_t tile_index, uint32_t group,
						     unsigned char *dynamic_shared, prefill_shared *shared)
{
	const prefill_tile_view tile = prefill_tile_of(record, arena, view, tile_index);
	const uint32_t H = record.input_size, I = prefill_inner_of(record, tile.tile.expert);
	const unsigned char *const matrices[2] = { arena + tile.gate, arena + tile.up };
	const uint64_t codes = exl3_code_bytes(H, I, BX2), first_scale = group * EXL3_TRANSFORM;
	prefill_fetch_scales(shared, 0u, reinterpret_cast<const __half *>(arena + tile.gate + codes) + H + first_scale);
	prefill_fetch_scales(shared, 1u, reinterpret_cast<const __half *>(arena + tile.up + codes) + H + first_scale);
	prefill_fetch_scales(shared, 2u, reinterpret_cast<const __half *>(arena + tile.down + exl3_code_bytes(I, H, BX2)) +
						 first_scale);
	prefill_thin_products<BX2, 2, 1>(matrices, I, group, 1u, view.workspace + view.parts.gate_up_operands +
					 (uint64_t)tile_index * H * 512u, tile.tile.row_count, H / EXL3_TILE, dynamic_shared);
	prefill_gate_up_rows(record, view, shared, tile, tile_index, 1u, group, reinterpret_cast<float *>(dynamic_shared));
}

/* down of such a tile by the groups first_group, + 1. Decode warps. */
template <uint32_t BX2>
__device__ __forceinline__ void prefill_thin_down(const struct exl3_prefill_record &record, unsigned char *arena,
						  const prefill_view &view, uint32_t tile_index, uint32_t first_group,
						  unsigned char *dynamic_shared, prefill_shared *shared)
{
	const prefill_tile_view tile = prefill_tile_of(record, arena, view, tile_index);
	const uint32_t H = record.input_size, I = prefill_inner_of(record, tile.tile.expert);
	const uint32_t groups = min(2u, H / EXL3_TRANSFORM - first_group);
	const unsigned char *const matrices[1] = { arena + tile.down };
	for (uint32_t g = 0; g < groups; g++)
		prefill_fetch_scales(shared, g, reinterpret_cast<const __half *>(arena + tile.down + exl3_code_bytes(I, H, BX2)) + I +
							 (first_group + g) * EXL3_TRANSFORM);
	prefill_thin_products<BX2, 1, 2>(matrices, H, first_group, groups, view.workspace + view.parts.down_operands +
					 (uint64_t)tile_index * view.widest * 256u, tile.tile.row_count, I / EXL3_TILE, dynamic_shared);
	prefill_down_rows(shared, tile, first_group, groups, H, reinterpret_cast<float *>(arena + record.pair_output_offset),
			  reinterpret_cast<const float *>(dynamic_shared));
}

#define PREFILL_WIDTH_SWITCH(call, otherwise)                                                          \
	switch (exl3_bits_x2(reinterpret_cast<const uint32_t *>(arena + record.widths_offset)[tile.expert])) { \
	case EXL3_BITS_X2_K2: {                                                                        \
		constexpr uint32_t BX2 = EXL3_BITS_X2_K2;                                              \
		call;                                                                                  \
	} break;                                                                                       \
	case EXL3_BITS_X2_K2_5: {                                                                      \
		constexpr uint32_t BX2 = EXL3_BITS_X2_K2_5;                                            \
		call;                                                                                  \
	} break;                                                                                       \
	case EXL3_BITS_X2_K3: {                                                                        \
		constexpr uint32_t BX2 = EXL3_BITS_X2_K3;                                              \
		call;                                                                                  \
	} break;                                                                                       \
	case EXL3_BITS_X2_K4: {                                                                        \
		constexpr uint32_t BX2 = EXL3_BITS_X2_K4;                                              \
		call;                                                                                  \
	} break;                                                                                       \
	default:                                                                                       \
		otherwise;                                                                             \
		break;                                                                                 \
	}

/* grid (ceil(widest I / 256), tile capacity) CTA pairs x 576 */
extern "C" __global__ void __cluster_dims__(PREFILL_PAIR, 1, 1) __launch_bounds__(EXL3_PREFILL_GEMM_THREADS, 1)
	exl3_prefill_gate_up(struct exl3_prefill_record record, unsigned char *arena)
{
	extern __shared__ __align__(1024) unsigned char dynamic_shared[];
	__shared__ prefill_shared shared;
	prefill_follow();
	const prefill_view view = prefill_view_of(record, arena);
	const uint32_t tile_count = reinterpret_cast<const uint32_t *>(view.workspace + view.parts.counts)[view.experts];
	if (blockIdx.y >= tile_count)
		return;
	/* the last tiles first: the always-on expert's, two to a unit, take half as long again as the median expert's */
	const uint32_t tile_index = tile_count - 1u - blockIdx.y;
	const uint32_t rank = blockIdx.x % PREFILL_PAIR, first_group = blockIdx.x / PREFILL_PAIR * 2u;
	const struct exl3_prefill_tile tile =
		reinterpret_cast<const struct exl3_prefill_tile *>(view.workspace + view.parts.tiles)[tile_index];
	const uint32_t count = prefill_tiles_of_unit(view, tile, tile_index, tile_count);
	if (count == 0 || first_group >= prefill_inner_of(record, tile.expert) / EXL3_TRANSFORM)
		return;
	if (count == 1u && tile.row_count <= PREFILL_THIN_ROWS) {
		if (threadIdx.x / EXL3_WARP >= PREFILL_FIRST_DECODE_WARP &&
		    first_group + rank < prefill_inner_of(record, tile.expert) / EXL3_TRANSFORM)
			PREFILL_WIDTH_SWITCH((prefill_thin_gate_up<BX2>(record, arena, view, tile_index, first_group + rank,
									dynamic_shared, &shared)), (void)0)
		return;
	}
	if (!prefill_begin(&shared, rank, prefill_rings<2, 1>::stages, prefill_rings<2, 1>::parts)) {
		prefill_release(&shared);
		return;
	}
	PREFILL_WIDTH_SWITCH((prefill_gate_up<BX2>(record, arena, view, tile_index, count, first_group + rank, rank, dynamic_shared,
						   &shared)), prefill_release(&shared))
}

/* grid (ceil(H / 512), tile capacity) CTA pairs x 576 */
extern "C" __global__ void __cluster_dims__(PREFILL_PAIR, 1, 1) __launch_bounds__(EXL3_PREFILL_GEMM_THREADS, 1)
	exl3_prefill_down(struct exl3_prefill_record record, unsigned char *arena)
{
	extern __shared__ __align__(1024) unsigned char dynamic_shared[];
	__shared__ prefill_shared shared;
	prefill_follow();
	const prefill_view view = prefill_view_of(record, arena);
	const uint32_t tile_count = reinterpret_cast<const uint32_t *>(view.workspace + view.parts.counts)[view.experts];
	if (blockIdx.y >= tile_count)
		return;
	/* the last tiles first: the always-on expert's, two to a unit, take half as long again as the median expert's */
	const uint32_t tile_index = tile_count - 1u - blockIdx.y;
	const uint32_t rank = blockIdx.x % PREFILL_PAIR, first_group = blockIdx.x / PREFILL_PAIR * 4u;
	const struct exl3_prefill_tile tile =
		reinterpret_cast<const struct exl3_prefill_tile *>(view.workspace + view.parts.tiles)[tile_index];
	const uint32_t count = prefill_tiles_of_unit(view, tile, tile_index, tile_count);
	if (count == 0)
		return;
	if (count == 1u && tile.row_count <= PREFILL_THIN_ROWS) {
		if (threadIdx.x / EXL3_WARP >= PREFILL_FIRST_DECODE_WARP && first_group + 2u * rank < record.input_size / EXL3_TRANSFORM)
			PREFILL_WIDTH_SWITCH((prefill_thin_down<BX2>(record, arena, view, tile_index, first_group + 2u * rank, dynamic_shared,
								     &shared)), (void)0)
		return;
	}
	if (!prefill_begin(&shared, rank, prefill_rings<1, 2>::stages, prefill_rings<1, 2>::parts)) {
		prefill_release(&shared);
		return;
	}
	PREFILL_WIDTH_SWITCH((prefill_down<BX2>(record, arena, view, tile_index, count, first_group + 2u * rank,
						min(2u, record.input_size / EXL3_TRANSFORM - first_group), rank, dynamic_shared,
						&shared)), prefill_release(&shared))
}

/* grid (ceil(H / 512), row capacity) x 128: FP32 row sums over the row's local pairs from +0 in ascending slot order,
 * four channels a thread */
extern "C" __global__ void __launch_bounds__(EXL3_ROW_SUM_THREADS)
	exl3_prefill_row_sum(struct exl3_prefill_record record, unsigned char *arena)
{
	const struct step_block step = *reinterpret_cast<const struct step_block *>(arena + record.step_offset);
	const uint32_t channel = (blockIdx.x * blockDim.x + threadIdx.x) * 4u;
	const uint64_t row = blockIdx.y;
	if (channel >= record.input_size || row >= min(step.row_count, record.row_capacity))
		return;
	const uint32_t width = record.input_size, slots = record.picks + record.shared_count;
	const float *const pairs = reinterpret_cast<const float *>(arena + record.pair_output_offset);
	const uint32_t *const picked = reinterpret_cast<const uint32_t *>(arena + record.picks_offset) + row * record.picks;
	float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
	for (uint32_t slot = 0; slot < slots; slot++) {
		/* a routed pair counts where its expert is held; an always-on pair everywhere it exists */
		if (slot < record.picks && picked[slot] - record.local_first >= record.local_count)
			continue;
		const float4 value = *reinterpret_cast<const float4 *>(pairs + (row * slots + slot) * width + channel);
		sum.x = __fadd_rn(sum.x, value.x);
		sum.y = __fadd_rn(sum.y, value.y);
		sum.z = __fadd_rn(sum.z, value.z);
		sum.w = __fadd_rn(sum.w, value.w);
	}
	*reinterpret_cast<float4 *>(reinterpret_cast<float *>(arena + record.row_output_offset) + row * width + channel) = sum;
}
