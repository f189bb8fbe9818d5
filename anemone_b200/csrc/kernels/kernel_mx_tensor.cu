/*
 * kernel_mx_tensor.cu: the original-weights layer's products on the fifth-generation tensor cores (struct
 * mx_products_arguments): MXFP4 routed experts and the E4M3 always-on expert by E4M3 block-quantized vectors, for a
 * decode step (mx_gate_up_few, mx_down_few) and for a prompt (mx_gate_up_many, mx_down_many). What bounds both is the
 * weights' way from HBM: an expert of a decode step sees a row or two, the median expert of a prompt a few. The weights
 * therefore stand in the operand of 128 rows of the block-scaled product (tcgen05.mma.kind::mxf8f6f4.block_scale, both
 * E8M0 scales applied by the tensor cores) and an expert's rows in its columns (16 to 128 of them): a weight costs a
 * quarter of an ALU instruction (its nibble moves to its place in the E2M1 operand, nothing is converted) and no
 * multiply-add.
 *
 * One persistent CTA a SM walks units: a tile of rows of one expert by 64 columns of gate and the same 64 of up (or
 * 128 outputs of down), all of K in stages of 256 inputs. Its warps:
 *   schedule  finds the CTA's units ahead of the others (matrices, rows, route weights) into a ring of eight
 *   weights   few: four teams of four warps, many: two teams of eight, that take the stages in turns; a lane keeps eight
 *             128-bit loads of its warp's tiles in flight in registers, across the units' ends, and stores a stage's
 *             codes as the A operand and its scales in the order tcgen05.cp takes them (no shared-memory copy of the raw words: the SM's
 *             shared-memory bandwidth is the next limit behind HBM). Teams because one warp's chain of wait,
 *             stores, fence and arrival is longer than a stage at the HBM rate (about 390 ns)
 *   rows      few: four warps, a stage each in turns, gather the rows' codes and exponents by cp.async as the B operand;
 *             many: one warp copies them in bulk from where mx_gather and the gate/up launch laid them in operand order
 *   multiply  one warp: scales to tensor memory, eight products of 32 inputs a stage, tcgen05.commit
 *   epilogue  the hidden step and its quantization (gate/up), or bfloat16 pair outputs (down)
 * The FP32 accumulators of two units alternate in tensor memory, so a unit's epilogue runs beside the next one's
 * products. The always-on expert with one FP32 scale per 128 x 128 weights takes the sum of every 128 inputs out of
 * tensor memory and adds it, times the scale, in FP32.
 * Every wait is bounded; one that runs out raises exl3_wait_expired, and the CTA ends without its remaining units.
 *
 * Measured (hidden 4096, intermediate 2048, 256 experts, top 8, CUDA events, one launch alone): eight rows, 508 MB of
 * gate and up in 116 us (4.4 TB/s; by two teams 127, the mma.sync launch 208), down 60 us (69, 115), the always-on expert
 * inside them (63 us of launches of its own before); 2048 rows, 867 + 444 us (6209 + 3337, and the always-on expert's 1415). Stages of 128
 * inputs, one team of weight warps or the products issued behind a lane test each made the multiplying or the weight
 * warps' chain the limit (246, 212 and 169 us at eight rows).
 */
#include "activation_quantize_device.cuh"
#include "exl3_device.cuh"

#include "anemone_b200_mx.h"

#define MX_THREADS MX_PRODUCTS_THREADS
#define MX_WARP_WEIGHTS 12u /* behind the epilogue's, the multiplying, the scheduling and the rows' warps */
#define MX_WEIGHT_WARPS 16u
#define MX_TILES 8u /* of 16 weight rows, of a unit */

#define MX_BLOCK_INPUTS 128u /* a block: the inputs whose scales one tcgen05.cp brings */
#define MX_STAGE_BLOCKS 2u
#define MX_PIECE 2048u /* bytes of 16 inputs of 128 operand rows */
#define MX_BLOCK_PIECES (MX_BLOCK_INPUTS / 16u)
#define MX_BLOCK (MX_BLOCK_PIECES * MX_PIECE)
#define MX_OPERAND (MX_STAGE_BLOCKS * MX_BLOCK)
#define MX_SCALE_BYTES 512u /* of 128 operand rows and a block */
#define MX_STAGE_SCALES (2u * MX_STAGE_BLOCKS * MX_SCALE_BYTES) /* [block][A, B] */

#define MX_UNIT_ROUTED 0u
#define MX_UNIT_SHARED 1u
#define MX_UNIT_END 2u
/* units the scheduler may be ahead: more than the units a warp's loads in flight can reach into (its team's next stage, or,
 * of eight warps, next two: four units where K is 256 or less), so that no role waits for a unit that waits for it */
#define MX_UNITS 8u
#define MX_CHUNK 4u /* loads of a lane stored, and asked for again, together; two chunks are in flight */
#define MX_SCALE_COLUMN 256u /* tensor memory: two accumulators of 128 columns, then the stages' scales */
#define MX_MOST_STAGES 5u

/* The two forms. FEW: units of a job table (at most eight rows, sixteen columns of the product). MANY: tiles of up to 128
 * rows whose vectors lie in operand order. */
template <bool FEW> struct mx_form {
	static constexpr uint32_t columns = FEW ? 16u : MX_TILE_ROWS; /* of the B operand in shared memory */
	static constexpr uint32_t piece = columns * 16u;
	static constexpr uint32_t b_operand = MX_STAGE_BLOCKS * MX_BLOCK_PIECES * piece;
	static constexpr uint32_t stages = FEW ? 5u : 3u;
	static constexpr uint32_t epilogue_warps = FEW ? 4u : 8u;
	static constexpr uint32_t row_warps = FEW ? 4u : 1u;
	/* The weights' warps in teams that take the stages in turns, each warp MX_TILES / team_warps tiles of its team's. What a
	 * stage costs a warp beside its stores (the wait for the place, the fence, the arrival, the next unit's pointers: about
	 * as much as one tile) is paid once for two tiles by teams of four, and four stages of the ring of five are filled at
	 * once (a call of eight rows 221 us by two teams of eight, 214 by four of four); the many rows' ring holds three. */
	static constexpr uint32_t team_warps = FEW ? 4u : 8u, teams = MX_WEIGHT_WARPS / team_warps;
	static constexpr uint32_t multiply = epilogue_warps, schedule = multiply + 1u, rows = schedule + 1u;
	static constexpr uint32_t b_at = stages * MX_OPERAND;
	static constexpr uint32_t scales_at = b_at + stages * b_operand;
	static constexpr uint32_t exchange_at = scales_at + stages * MX_STAGE_SCALES; /* two turns of a warp's eight columns */
	static constexpr uint32_t codes_at = exchange_at + 2u * epilogue_warps * 8u * 32u * 4u;
	static constexpr uint32_t bytes = codes_at + epilogue_warps * 8u * 32u;
	static_assert(bytes <= MX_PRODUCTS_DYNAMIC_BYTES && stages <= MX_MOST_STAGES, "the host sizes the shared memory");
	static_assert(rows + row_warps <= MX_WARP_WEIGHTS, "the warps' order");
};
static_assert((MX_WARP_WEIGHTS + MX_WEIGHT_WARPS) * EXL3_WARP == MX_THREADS, "the warps of a CTA");

struct mx_unit {
	const unsigned char *matrix[2];
	const unsigned char *b_codes, *b_scales; /* MANY: the tile's vectors in operand order */
	uint32_t kind;
	uint32_t rows;
	uint32_t group; /* of 64 columns of gate and up, or of 128 outputs of down */
	uint32_t tile; /* MANY: the operand-order tile */
	uint32_t vector[MX_TILE_ROWS]; /* pair, or row of the always-on expert */
	float weight[MX_TILE_ROWS];
};

struct mx_shared {
	struct mx_unit units[MX_UNITS];
	uint64_t unit_full[MX_UNITS], unit_free[MX_UNITS];
	uint64_t full[MX_MOST_STAGES], empty[MX_MOST_STAGES];
	uint64_t sum_full[2], sum_free[2];
	uint64_t done;
	uint32_t tensor_memory;
};

/* ------------------------------------------------------------------ tensor-core instructions */

/* Shared-memory descriptors in two words, the second constant. Operands: no swizzle, K-major, 16-byte pieces of eight
 * rows adjacent, the groups of eight rows adjacent, `piece` to the next sixteen inputs. Scales: 32 rows of 16 bytes. */
#define MX_DESCRIPTOR_HIGH ((128u >> 4) | 1u << 14)
__device__ __forceinline__ uint32_t mx_operand_descriptor(uint32_t shared_address, uint32_t piece)
{
	return shared_address >> 4 | (piece >> 4) << 16;
}

__device__ __forceinline__ uint32_t mx_scale_descriptor(uint32_t shared_address)
{
	return shared_address >> 4 | (128u >> 4) << 16;
}

/* A of E2M1 (5) or E4M3 (0), B of E4M3, E8M0 scales, FP32 accumulators, M = 128, N = columns */
__device__ __forceinline__ uint32_t mx_instruction(uint32_t a_format, uint32_t columns)
{
	return a_format << 7 | (columns >> 3) << 17 | 1u << 23 | 1u << 27;
}

__device__ __forceinline__ void mx_scales_to_tensor_memory(uint32_t column, uint32_t descriptor)
{
	asm volatile("{\n\t.reg .b64 d;\n\t"
		     "mov.b64 d, {%1, %2};\n\t"
		     "tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], d;\n\t}" ::"r"(column),
		     "r"(descriptor), "n"(MX_DESCRIPTOR_HIGH)
		     : "memory");
}

/* a_scales, b_scales: tensor-memory columns, multiples of four (a unit's rows always begin at its scales' first) */
__device__ __forceinline__ void mx_multiply(uint32_t sums, uint32_t a, uint32_t b, uint32_t instruction, uint32_t a_scales,
					    uint32_t b_scales, uint32_t accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
		     "setp.ne.b32 p, %6, 0;\n\t"
		     "mov.b64 a, {%1, %7};\n\t"
		     "mov.b64 b, {%2, %7};\n\t"
		     "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], a, b, %3, [%4], [%5], p;\n\t}" ::"r"(
			     sums),
		     "r"(a), "r"(b), "r"(instruction), "r"(a_scales), "r"(b_scales), "r"(accumulate), "n"(MX_DESCRIPTOR_HIGH)
		     : "memory");
}

__device__ __forceinline__ void mx_commit(uint64_t *barrier)
{
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_address(barrier))
		     : "memory");
}

/* one lane of the warp, the same one every time */
__device__ __forceinline__ bool mx_elected()
{
	uint32_t elected;
	asm volatile("{\n\t.reg .pred p;\n\t"
		     "elect.sync _|p, 0xFFFFFFFF;\n\t"
		     "selp.u32 %0, 1, 0, p;\n\t}"
		     : "=r"(elected));
	return elected != 0;
}

__device__ __forceinline__ void mx_fence_before()
{
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void mx_fence_after()
{
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void mx_proxy_fence()
{
	asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

/* sixteen columns of this warp's quarter of the accumulator rows, a row a lane */
__device__ __forceinline__ void mx_load_sums(uint32_t address, float out[16])
{
	uint32_t r[16];
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
		     "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
		     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
		       "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
		     : "r"(address)
		     : "memory");
	asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
	for (uint32_t i = 0; i < 16; i++)
		out[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t mx_bfloat16_bits(float value)
{
	const uint32_t bits = __float_as_uint(value);
	return (bits & 0x7FFFFFFFu) > 0x7F800000u ? 0x7FC0u : (bits + 0x7FFFu + ((bits >> 16) & 1u)) >> 16;
}

/* A whole warp's wait: its lanes go on, or give up, together. */
__device__ __forceinline__ bool mx_wait(uint64_t *barrier, uint32_t parity)
{
	return __all_sync(0xFFFFFFFFu, barrier_wait(barrier, parity)) != 0;
}

/* The epilogue warps' verdicts together: true where every one of them may go on (they meet at named barriers, so none
 * may leave alone). */
template <uint32_t WARPS> __device__ __forceinline__ bool mx_agree(bool good)
{
	uint32_t all;
	asm volatile("{\n\t.reg .pred p, q;\n\t"
		     "setp.ne.b32 p, %1, 0;\n\t"
		     "barrier.cta.red.and.pred q, 7, %2, p;\n\t"
		     "selp.u32 %0, 1, 0, q;\n\t}"
		     : "=r"(all)
		     : "r"(good ? 1u : 0u), "n"(WARPS * EXL3_WARP)
		     : "memory");
	return all != 0;
}

/* ------------------------------------------------------------------ the rings */

/* A role's place in the ring of units. */
struct mx_place {
	uint32_t next;
	__device__ __forceinline__ const struct mx_unit *peek(struct mx_shared &shared) const
	{
		return mx_wait(&shared.unit_full[next % MX_UNITS], (next / MX_UNITS) & 1u) ? &shared.units[next % MX_UNITS] :
											       nullptr;
	}
	__device__ __forceinline__ void release(struct mx_shared &shared, uint32_t lane)
	{
		__syncwarp();
		if (lane == 0)
			barrier_arrive(&shared.unit_free[next % MX_UNITS]);
		next++;
	}
};

/* A role's place in the ring of stages: the slot and the parity of its turn. */
template <uint32_t STAGES> struct mx_stage_place {
	uint32_t slot, parity;
	__device__ __forceinline__ void advance(uint32_t step)
	{
		slot += step;
		if (slot >= STAGES) {
			slot -= STAGES;
			parity ^= 1u;
		}
	}
};

__device__ __forceinline__ uint32_t mx_stages_of(uint32_t inputs)
{
	return (inputs / MX_BLOCK_INPUTS + MX_STAGE_BLOCKS - 1u) / MX_STAGE_BLOCKS;
}

template <bool DOWN, bool FEW>
__device__ __forceinline__ void mx_schedule(const struct mx_products_arguments &arguments, unsigned char *arena,
					    struct mx_shared &shared, uint32_t lane)
{
	const struct step_block step = *reinterpret_cast<const struct step_block *>(arena + arguments.step_offset);
	const uint32_t live = min(step.row_count, arguments.row_capacity), K = arguments.input_size;
	const uint32_t groups = arguments.output_size / (DOWN ? 128u : 64u);
	const uint32_t shared_rows = mx_shared_tile_rows(arguments.shared_format);
	const uint32_t shared_units =
		arguments.shared_format == MX_SHARED_NONE ? 0u : (live + shared_rows - 1u) / shared_rows * groups;
	const uint32_t tiles =
		FEW ? arguments.tile_capacity :
		      min(reinterpret_cast<const uint32_t *>(arena + arguments.counts_offset)[arguments.expert_count],
			  arguments.tile_capacity);
	for (uint32_t index = blockIdx.x, turn = 0;; index += gridDim.x, turn++) {
		const uint32_t slot = turn % MX_UNITS, use = turn / MX_UNITS;
		if (use > 0 && !mx_wait(&shared.unit_free[slot], (use - 1u) & 1u))
			return;
		struct mx_unit *const unit = &shared.units[slot];
		uint32_t kind = MX_UNIT_END, rows = 0, group = 0, tile = 0;
		const unsigned char *first = nullptr, *second = nullptr;
		if (index < shared_units) {
			const uint32_t base = index / groups * shared_rows;
			kind = MX_UNIT_SHARED;
			group = index % groups;
			rows = min(live - base, shared_rows);
			tile = arguments.tile_capacity + base / shared_rows;
			first = arena + arguments.shared_weights_offset[0];
			second = arena + arguments.shared_weights_offset[1];
			for (uint32_t row = lane; row < rows; row += EXL3_WARP) {
				unit->vector[row] = base + row;
				unit->weight[row] = 1.0f;
			}
		} else {
			tile = (index - shared_units) / groups;
			group = (index - shared_units) % groups;
			if (FEW && tile < tiles) {
				const struct expert_job_record *const job =
					reinterpret_cast<const struct expert_job_record *>(arena + arguments.jobs_offset) + tile;
				rows = job->row_count;
				if (rows != 0) { /* the live jobs stand in front */
					kind = MX_UNIT_ROUTED;
					first = arena + (DOWN ? job->down_offset : job->gate_offset);
					second = arena + job->up_offset;
					if (lane < rows) {
						unit->vector[lane] = job->pair_index[lane];
						unit->weight[lane] = job->route_weight[lane];
					}
				}
			} else if (!FEW && tile < tiles) {
				const struct exl3_prefill_tile record =
					reinterpret_cast<const struct exl3_prefill_tile *>(arena + arguments.tiles_offset)[tile];
				const uint64_t *const table =
					reinterpret_cast<const uint64_t *>(arena + arguments.expert_table_offset) + 3u * record.expert;
				const struct exl3_prefill_entry *const entries =
					reinterpret_cast<const struct exl3_prefill_entry *>(arena + arguments.entries_offset) +
					(uint64_t)record.expert * arguments.row_capacity + record.first_entry;
				kind = MX_UNIT_ROUTED;
				rows = record.row_count;
				first = arena + table[DOWN ? 2 : 0];
				second = arena + table[1];
				for (uint32_t row = lane; row < rows; row += EXL3_WARP) {
					const struct exl3_prefill_entry entry = entries[row];
					unit->vector[row] = entry.pair;
					unit->weight[row] = entry.route_weight;
				}
			}
		}
		if (lane == 0) {
			unit->matrix[0] = first;
			unit->matrix[1] = DOWN ? first : second;
			unit->b_codes = arena + arguments.codes_offset + (uint64_t)tile * MX_TILE_ROWS * K;
			unit->b_scales = arena + arguments.exponents_offset +
					 (uint64_t)tile * (K / MX_BLOCK_INPUTS) * MX_SCALE_BYTES;
			unit->kind = kind;
			unit->rows = rows;
			unit->group = group;
			unit->tile = tile;
		}
		__syncwarp();
		if (lane == 0)
			barrier_arrive(&shared.unit_full[slot]);
		if (kind == MX_UNIT_END)
			return;
	}
}

/* ------------------------------------------------------------------ weights */

/* A stored load of 16 outputs x 64 MXFP4 inputs (a lane's four words: outputs g and g + 8, two blocks of 32) into the
 * operand: 16 E2M1 codes stand in the first eight of their sixteen bytes */
__device__ __forceinline__ void mx_store_nibbles(unsigned char *to, const uint4 &words)
{
	const uint32_t low = 0x0F0F0F0Fu;
	*reinterpret_cast<uint32_t *>(to) = (words.x & low) | ((words.y << 4) & ~low);
	*reinterpret_cast<uint32_t *>(to + 128u) = ((words.x >> 4) & low) | (words.y & ~low);
	*reinterpret_cast<uint32_t *>(to + 2u * MX_PIECE) = (words.z & low) | ((words.w << 4) & ~low);
	*reinterpret_cast<uint32_t *>(to + 2u * MX_PIECE + 128u) = ((words.z >> 4) & low) | (words.w & ~low);
}

/* A stored group of 16 outputs x 32 E4M3 inputs into the operand */
__device__ __forceinline__ void mx_store_bytes(unsigned char *to, const uint4 &words)
{
	uint32_t first = __byte_perm(words.x, words.z, 0x6240), second = __byte_perm(words.y, words.w, 0x6240);
	*reinterpret_cast<uint2 *>(to) = make_uint2(__byte_perm(first, second, 0x5410), __byte_perm(first, second, 0x7632));
	first = __byte_perm(words.x, words.z, 0x7351), second = __byte_perm(words.y, words.w, 0x7351);
	*reinterpret_cast<uint2 *>(to + 128u) =
		make_uint2(__byte_perm(first, second, 0x5410), __byte_perm(first, second, 0x7632));
}

/* The scales of a tile of 16 weight rows and a stage, where tcgen05.cp takes them: byte 4 (r / 32) + b of the sixteen of
 * row r % 32 is the scale of block b of 32 inputs. MXFP4: lane 8 l + g holds the word of load l of 64 inputs and of rows
 * g and g + 8. E4M3: lane 16 b + r holds the four codes of row r and of block b of 128 inputs. */
template <bool BYTES> __device__ __forceinline__ void mx_store_scales(unsigned char *to, uint32_t word)
{
	if (BYTES) {
		*reinterpret_cast<uint32_t *>(to) = word;
	} else {
		*reinterpret_cast<uint16_t *>(to) = (uint16_t)__byte_perm(word, 0, 0x4420);
		*reinterpret_cast<uint16_t *>(to + 128u) = (uint16_t)__byte_perm(word, 0, 0x4431);
	}
}

template <uint32_t STAGES> struct mx_weights_place {
	struct mx_place units;
	struct mx_stage_place<STAGES> stage;
	uint32_t begun; /* stages of the units entered so far: they say whose the next unit's first stage is */
};

/* The units of one kind that follow one another, by one warp of a team: its tiles of 16 weight rows of every stage of its
 * team's. A stage is a run of chunks of MX_CHUNK loads (MXFP4: a tile; E4M3: half a tile, a block); a chunk's registers are
 * asked for the chunk after next as soon as they are stored, across the stages' and the units' ends. False once a wait ran
 * out. */
template <bool DOWN, bool FEW, bool BYTES>
__device__ __forceinline__ bool mx_weights(const struct mx_products_arguments &arguments, const unsigned char *arena,
					   struct mx_shared &shared, unsigned char *dynamic_shared, uint32_t lane, uint32_t team,
					   uint32_t warp, struct mx_weights_place<mx_form<FEW>::stages> &place)
{
	typedef mx_form<FEW> form;
	constexpr uint32_t kind = BYTES ? MX_UNIT_SHARED : MX_UNIT_ROUTED;
	constexpr uint32_t tiles = MX_TILES / form::team_warps, halves = BYTES ? 2u : 1u, chunks = tiles * halves;
	constexpr uint32_t block_items = BYTES ? 4u : 2u, stage_items = MX_STAGE_BLOCKS * block_items; /* of a tile */
	constexpr uint32_t turn = chunks < 2u ? 2u : chunks; /* chunks of one turn of the loop */
	static_assert(halves * MX_CHUNK == stage_items && turn % 2u == 0u && turn % chunks == 0u, "chunks make stages");
	const uint32_t K = arguments.input_size, blocks = K / MX_BLOCK_INPUTS, stages = mx_stages_of(K);
	const uint64_t weights = (uint64_t)arguments.output_size * K;
	const bool constant_scales = BYTES && arguments.shared_format == WEIGHT_FORMAT_E4M3_BLOCK128;
	uint4 held[2][MX_CHUNK];
	uint32_t scales[2];
	const uint4 *from[tiles]; /* of the stage whose chunks are asked for */
	const uint32_t *scales_from[tiles];
	uint32_t at = stages, pending = 0; /* at: that stage of its unit; from `stages` on: the unit has no more */
	bool more = true, good = true;
#pragma unroll
	for (uint32_t tile = 0; tile < tiles; tile++) {
		from[tile] = reinterpret_cast<const uint4 *>(arena);
		scales_from[tile] = reinterpret_cast<const uint32_t *>(arena);
	}
	/* the next stage of the team's, in this unit or one behind it */
	auto enter = [&]() {
		if (more) {
			at += form::teams;
#pragma unroll
			for (uint32_t tile = 0; tile < tiles; tile++) {
				from[tile] += form::teams * stage_items * EXL3_WARP;
				scales_from[tile] += form::teams * MX_STAGE_BLOCKS * (BYTES ? 1u : 16u);
			}
		}
		while (more && at >= stages) {
			const struct mx_unit *const unit = place.units.peek(shared);
			good = unit != nullptr;
			more = good && unit->kind == kind;
			if (more) {
				at = (team - place.begun) % form::teams;
				place.begun += stages;
#pragma unroll
				for (uint32_t tile = 0; tile < tiles; tile++) {
					const uint32_t local = tile * form::team_warps + warp;
					const uint32_t row_tile = DOWN ? unit->group * 8u + local : unit->group * 4u + local % 4u;
					const unsigned char *const matrix = unit->matrix[DOWN ? 0u : local / 4u];
					from[tile] = reinterpret_cast<const uint4 *>(matrix) +
						     ((uint64_t)row_tile * blocks + at * MX_STAGE_BLOCKS) * (block_items * EXL3_WARP) + lane;
					if (BYTES)
						scales_from[tile] = reinterpret_cast<const uint32_t *>(
									    matrix + weights + (uint64_t)(row_tile / 2u) * (K / 32u)) +
								    at * MX_STAGE_BLOCKS + lane / 16u;
					else
						scales_from[tile] = reinterpret_cast<const uint32_t *>(matrix + weights / 2u) +
								    ((uint64_t)row_tile * blocks + at * MX_STAGE_BLOCKS) * 16u + lane;
				}
				place.units.release(shared, lane);
			}
		}
		pending += more ? 1u : 0u;
	};
	/* Chunk `sub` of that stage into place `to`. Every register is loaded on every path (the arena's first bytes where there
	 * is no stage left; a last stage of one block brings its first block twice, and nothing reads the second's place): a
	 * load under a condition would make a copy of the register where the paths meet, and the copy waits for the load. */
	auto ask = [&](uint32_t to, uint32_t sub) {
		const uint32_t tile = sub / halves, half = sub % halves;
		const bool whole = at * MX_STAGE_BLOCKS + 1u < blocks;
		const uint4 *const first = more ? from[tile] : reinterpret_cast<const uint4 *>(arena);
		const uint32_t step = more ? EXL3_WARP : 0u, second = more && whole ? block_items * EXL3_WARP : 0u;
#pragma unroll
		for (uint32_t item = 0; item < MX_CHUNK; item++) {
			const uint32_t stage_item = half * MX_CHUNK + item;
			held[to][item] = __ldcs(first + stage_item % block_items * step + (stage_item < block_items ? 0u : second));
		}
		if (half == 0u)
			scales[to] = __ldg(more && !constant_scales ?
						   scales_from[tile] - (whole || lane < 16u ? 0u : BYTES ? 1u : 16u) :
						   reinterpret_cast<const uint32_t *>(arena));
	};
	enter();
	ask(0u, 0u);
	if (chunks == 1u)
		enter();
	ask(1u, 1u % chunks);
	/* lane 4 g + t: row g of the tile, its quarter t of the block's inputs */
	unsigned char *const lane_at = dynamic_shared + (lane % 4u / 2u) * MX_PIECE + (warp * 16u + lane / 4u) * 16u +
				       (lane % 2u) * (BYTES ? 8u : 4u);
	const uint32_t row = warp * 16u + (BYTES ? lane % 16u : lane % 8u);
	unsigned char *const lane_scales = dynamic_shared + form::scales_at + row % 32u * 16u + row / 32u * 4u +
					   lane / 16u * (2u * MX_SCALE_BYTES) + (BYTES ? 0u : lane / 8u % 2u * 2u);
	while (good && pending != 0) {
#pragma unroll
		for (uint32_t chunk = 0; chunk < turn; chunk++) {
			const uint32_t sub = chunk % chunks, tile = sub / halves, half = sub % halves, here = chunk % 2u;
			if (sub == 0u) {
				if (!good || pending == 0)
					break;
				good = mx_wait(&shared.empty[place.stage.slot], place.stage.parity ^ 1u);
			}
			unsigned char *const to = lane_at + place.stage.slot * MX_OPERAND + tile * (form::team_warps * 256u);
#pragma unroll
			for (uint32_t item = 0; item < MX_CHUNK; item++)
				if (BYTES)
					mx_store_bytes(to + (half * MX_CHUNK + item) * 2u * MX_PIECE, held[here][item]);
				else
					mx_store_nibbles(to + item * 4u * MX_PIECE, held[here][item]);
			if (half == 0u)
				mx_store_scales<BYTES>(lane_scales + place.stage.slot * MX_STAGE_SCALES + tile * (form::team_warps / 2u * 4u),
						       constant_scales ? 0x7F7F7F7Fu : scales[here]);
			if (sub == chunks - 1u) {
				mx_proxy_fence();
				__syncwarp();
				if (lane == 0)
					barrier_arrive(&shared.full[place.stage.slot]);
				place.stage.advance(form::teams);
				pending--;
			}
			more = more && good;
			if ((chunk + 2u) % chunks == 0u)
				enter();
			ask(here, (chunk + 2u) % chunks);
		}
	}
	return good;
}

/* ------------------------------------------------------------------ the rows */

/* FEW: warp w of four takes every fourth stage. Two lanes a row (adjacent pieces: a whole sector of the row); a lane a
 * row's scales. The rows of a decode step lie in L2: a stage's copies have landed about a stage's turn later. */
template <bool DOWN>
__device__ __forceinline__ void mx_rows_few(const struct mx_products_arguments &arguments, const unsigned char *arena,
					    struct mx_shared &shared, unsigned char *dynamic_shared, uint32_t lane, uint32_t warp)
{
	typedef mx_form<true> form;
	const uint32_t K = arguments.input_size, blocks = K / MX_BLOCK_INPUTS, stages = mx_stages_of(K);
	struct mx_place place = { 0 };
	struct mx_stage_place<form::stages> stage = { warp, 0u };
	const uint32_t half = lane % 2u, row = lane / 2u;
	const uint32_t lane_at = smem_address(dynamic_shared) + form::b_at + half * form::piece + row * 16u;
	const uint32_t scales_at = smem_address(dynamic_shared) + form::scales_at + MX_SCALE_BYTES + lane * 16u;
	uint32_t begun = 0;
	for (;;) {
		const struct mx_unit *const unit = place.peek(shared);
		if (unit == nullptr)
			return;
		const uint32_t kind = unit->kind, rows = unit->rows;
		if (kind == MX_UNIT_END)
			return;
		const uint32_t first = (warp - begun) % form::row_warps;
		begun += stages;
		const uint32_t divisor = DOWN || kind == MX_UNIT_SHARED ? 1u : arguments.pairs_per_row;
		const unsigned char *const codes =
			arena + (kind == MX_UNIT_SHARED ? arguments.shared_codes_offset : arguments.codes_offset) + half * 16u;
		const unsigned char *const exponents =
			arena + (kind == MX_UNIT_SHARED ? arguments.shared_exponents_offset : arguments.exponents_offset);
		const unsigned char *const from = codes + (uint64_t)(row < rows ? unit->vector[row] / divisor : 0u) * K;
		const unsigned char *const scales =
			exponents + (uint64_t)(lane < rows ? unit->vector[lane] / divisor : 0u) * (K / 32u);
		place.release(shared, lane);
		for (uint32_t s = first; s < stages; s += form::row_warps) {
			if (!mx_wait(&shared.empty[stage.slot], stage.parity ^ 1u))
				return;
			const bool whole = s * MX_STAGE_BLOCKS + 1u < blocks;
			if (row < rows) {
#pragma unroll
				for (uint32_t pair = 0; pair < MX_STAGE_BLOCKS * MX_BLOCK_PIECES / 2u; pair++)
					if (pair < MX_BLOCK_PIECES / 2u || whole)
						asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
								     lane_at + stage.slot * form::b_operand + pair * 2u * form::piece),
							     "l"(from + s * (MX_STAGE_BLOCKS * MX_BLOCK_INPUTS) + pair * 32u)
							     : "memory");
			}
			if (lane < rows) {
#pragma unroll
				for (uint32_t b = 0; b < MX_STAGE_BLOCKS; b++)
					if (b == 0 || whole)
						asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
								     scales_at + stage.slot * MX_STAGE_SCALES + b * 2u * MX_SCALE_BYTES),
							     "l"(scales + (s * MX_STAGE_BLOCKS + b) * 4u)
							     : "memory");
			}
			asm volatile("cp.async.wait_all;" ::: "memory");
			mx_proxy_fence();
			__syncwarp();
			if (lane == 0)
				barrier_arrive(&shared.full[stage.slot]);
			stage.advance(form::row_warps);
		}
	}
}

/* MANY: a stage's rows lie in operand order: a piece of 16 inputs (all pieces at once where the tile is full) and a
 * block's scales are each one bulk copy. */
__device__ __forceinline__ void mx_rows_many(const struct mx_products_arguments &arguments, struct mx_shared &shared,
					     unsigned char *dynamic_shared, uint32_t lane)
{
	typedef mx_form<false> form;
	const uint32_t blocks = arguments.input_size / MX_BLOCK_INPUTS, stages = mx_stages_of(arguments.input_size);
	struct mx_place place = { 0 };
	struct mx_stage_place<form::stages> stage = { 0u, 0u };
	for (;;) {
		const struct mx_unit *const unit = place.peek(shared);
		if (unit == nullptr || unit->kind == MX_UNIT_END)
			return;
		const uint32_t row_bytes = (unit->rows + 15u) / 16u * 256u;
		const unsigned char *codes = unit->b_codes + lane * MX_PIECE, *scales = unit->b_scales + lane * MX_SCALE_BYTES;
		place.release(shared, lane);
		for (uint32_t s = 0; s < stages; s++) {
			const uint32_t stage_blocks = min(blocks - s * MX_STAGE_BLOCKS, MX_STAGE_BLOCKS);
			const uint32_t pieces = stage_blocks * MX_BLOCK_PIECES;
			if (!mx_wait(&shared.empty[stage.slot], stage.parity ^ 1u))
				return;
			uint64_t *const full = &shared.full[stage.slot];
			if (lane == 0)
				barrier_expect(full, pieces * row_bytes + stage_blocks * MX_SCALE_BYTES);
			__syncwarp();
			unsigned char *const to = dynamic_shared + form::b_at + stage.slot * form::b_operand + lane * MX_PIECE;
			if (row_bytes == MX_PIECE) {
				if (lane == 0)
					bulk_load(to, codes, pieces * MX_PIECE, full);
			} else if (lane < pieces) {
				bulk_load(to, codes, row_bytes, full);
			}
			if (lane < stage_blocks)
				bulk_load(dynamic_shared + form::scales_at + stage.slot * MX_STAGE_SCALES +
						  lane * 2u * MX_SCALE_BYTES + MX_SCALE_BYTES,
					  scales, MX_SCALE_BYTES, full);
			codes += MX_STAGE_BLOCKS * MX_BLOCK;
			scales += MX_STAGE_BLOCKS * MX_SCALE_BYTES;
			stage.advance(1u);
		}
	}
}

/* ------------------------------------------------------------------ the products */

/* one block of 128 inputs: scales to tensor memory, four products */
template <uint32_t PIECE>
__device__ __forceinline__ void mx_block(uint32_t sums, uint32_t a, uint32_t b, uint32_t instruction, uint32_t scales,
					 uint32_t scale_column, bool first)
{
	mx_scales_to_tensor_memory(scale_column, scales);
	mx_scales_to_tensor_memory(scale_column + 4u, scales + (MX_SCALE_BYTES >> 4));
	mx_multiply(sums, a, b, instruction, scale_column, scale_column + 4u, first ? 0u : 1u);
#pragma unroll
	for (uint32_t k = 1; k < 4u; k++)
		mx_multiply(sums, a + k * (2u * MX_PIECE >> 4), b + k * (2u * PIECE >> 4), instruction + k * (1u << 4 | 1u << 29),
			    scale_column, scale_column + 4u, 1u);
}

/* The whole warp walks the stages (what it computes then lives in the warp's uniform registers, where the products want
 * it), one elected lane issues. */
template <bool FEW>
__device__ __forceinline__ void mx_products(const struct mx_products_arguments &arguments, struct mx_shared &shared,
					    unsigned char *dynamic_shared, uint32_t lane)
{
	typedef mx_form<FEW> form;
	const uint32_t blocks = arguments.input_size / MX_BLOCK_INPUTS, stages = mx_stages_of(arguments.input_size);
	const uint32_t tensor_memory = __shfl_sync(0xFFFFFFFFu, shared.tensor_memory, 0);
	const bool block128 = arguments.shared_format == WEIGHT_FORMAT_E4M3_BLOCK128;
	const uint32_t first_a = mx_operand_descriptor(smem_address(dynamic_shared), MX_PIECE);
	const uint32_t first_b = mx_operand_descriptor(smem_address(dynamic_shared + form::b_at), form::piece);
	const uint32_t first_scales = mx_scale_descriptor(smem_address(dynamic_shared + form::scales_at));
	struct mx_place place = { 0 };
	struct mx_stage_place<form::stages> stage = { 0u, 0u };
	uint32_t sum = 0, sum_parity = 0; /* the accumulator in turn, and the parity of its turn */
#define MX_NEXT_SUM()                   \
	do {                            \
		sum ^= 1u;              \
		sum_parity ^= sum ^ 1u; \
	} while (0)
	bool good = true;
	while (good) {
		const struct mx_unit *const unit = place.peek(shared);
		if (unit == nullptr)
			break;
		const uint32_t kind = __shfl_sync(0xFFFFFFFFu, unit->kind, 0);
		if (kind == MX_UNIT_END)
			break;
		const uint32_t columns = (__shfl_sync(0xFFFFFFFFu, unit->rows, 0) + 15u) / 16u * 16u;
		const uint32_t instruction = mx_instruction(kind == MX_UNIT_SHARED ? 0u : 5u, columns);
		place.release(shared, lane);
		const bool apart = kind == MX_UNIT_SHARED && block128; /* every block a sum of its own */
		if (!apart)
			good = mx_wait(&shared.sum_free[sum], sum_parity ^ 1u);
		for (uint32_t s = 0; s < stages && good; s++) {
			good = mx_wait(&shared.full[stage.slot], stage.parity);
			if (!good)
				break;
			mx_fence_after();
			const bool whole = s * MX_STAGE_BLOCKS + 1u < blocks;
			const uint32_t scales = first_scales + stage.slot * (MX_STAGE_SCALES >> 4);
			const uint32_t column = tensor_memory + MX_SCALE_COLUMN + stage.slot * (MX_STAGE_BLOCKS * 8u);
			const uint32_t a = first_a + stage.slot * (MX_OPERAND >> 4), b = first_b + stage.slot * (form::b_operand >> 4);
			if (apart) {
				for (uint32_t half = 0; half < (whole ? 2u : 1u) && good; half++) {
					good = mx_wait(&shared.sum_free[sum], sum_parity ^ 1u);
					if (!good)
						break;
					mx_fence_after();
					if (mx_elected()) {
						mx_block<form::piece>(tensor_memory + sum * 128u, a + half * (MX_BLOCK >> 4),
								      b + half * (MX_BLOCK_PIECES * form::piece >> 4), instruction,
								      scales + half * (2u * MX_SCALE_BYTES >> 4), column + half * 8u, true);
						mx_commit(&shared.sum_full[sum]);
					}
					__syncwarp();
					MX_NEXT_SUM();
				}
				if (good && mx_elected())
					mx_commit(&shared.empty[stage.slot]);
			} else if (mx_elected()) {
				mx_block<form::piece>(tensor_memory + sum * 128u, a, b, instruction, scales, column, s == 0);
				if (whole)
					mx_block<form::piece>(tensor_memory + sum * 128u, a + (MX_BLOCK >> 4),
							      b + (MX_BLOCK_PIECES * form::piece >> 4), instruction,
							      scales + (2u * MX_SCALE_BYTES >> 4), column + 8u, false);
				mx_commit(&shared.empty[stage.slot]);
				if (s + 1u == stages)
					mx_commit(&shared.sum_full[sum]);
			}
			__syncwarp();
			stage.advance(1u);
		}
		if (!apart)
			MX_NEXT_SUM();
	}
#undef MX_NEXT_SUM
	/* every product is done before the tensor memory is freed (the lane that issued them commits) */
	if (mx_elected())
		mx_commit(&shared.done);
	__syncwarp();
	(void)mx_wait(&shared.done, 0u);
}

/* ------------------------------------------------------------------ epilogues */

/* Sixteen columns (rows of the batch) of a gate/up unit: of four warps the first two hold gate's columns 0..31 and
 * 32..63 of the 64, the others up's. Warps w and w + 2 exchange halves, so that each forms the hidden values of eight
 * rows; a lane an output, a warp a block of 32 of the hidden vector's quantization. turn: counts the warp's calls. */
template <bool FEW>
__device__ __forceinline__ void mx_hidden(const struct mx_products_arguments &arguments, unsigned char *arena,
					  const struct mx_unit *unit, unsigned char *dynamic_shared, const float sums[16],
					  uint32_t chunk, uint32_t turn, uint32_t lane, uint32_t warp)
{
	typedef mx_form<FEW> form;
	const uint32_t q = warp % 2u;
	const bool is_up = warp % 4u >= 2u;
	float value[16];
#pragma unroll
	for (uint32_t i = 0; i < 16; i++) /* gate and up are bfloat16 first, as the reference's linear returns them */
		value[i] = __uint_as_float(mx_bfloat16_bits(sums[i]) << 16);
	float *const exchange = reinterpret_cast<float *>(dynamic_shared + form::exchange_at) +
				turn % 2u * (form::epilogue_warps * 256u) + lane;
#pragma unroll
	for (uint32_t i = 0; i < 8; i++)
		exchange[warp * 256u + i * 32u] = is_up ? value[i] : value[8u + i];
	asm volatile("bar.sync %0, 64;" ::"r"(1u + warp / 4u * 2u + q) : "memory");
	const uint32_t first = chunk * 16u + (is_up ? 8u : 0u);
	const float limit = arguments.activation_limit;
	unsigned char *const codes = dynamic_shared + form::codes_at + warp * 256u;
	/* where this lane's output stands in its block: value 16 p + k, k = 2 t + h + 8 r */
	const uint32_t k = lane % 16u, at = (k % 8u / 2u) * 8u + (2u * (k % 2u) + k / 8u) * 2u + lane / 16u;
	uint32_t exponent = 0;
#pragma unroll
	for (uint32_t i = 0; i < 8; i += 2) {
		float hidden[2];
		uint32_t sign[2];
#pragma unroll
		for (uint32_t j = 0; j < 2; j++) {
			const float other = exchange[(warp ^ 2u) * 256u + (i + j) * 32u];
			const float g = is_up ? other : value[i + j], u = is_up ? value[8u + i + j] : other;
			const float bounded_gate = g > limit ? limit : g;
			const float bounded_up = u > limit ? limit : (u < -limit ? -limit : u);
			const float gated = __fdiv_rn(bounded_gate, __fadd_rn(1.0f, expf(-bounded_gate)));
			const uint32_t column = first + i + j;
			const float weight = column < unit->rows ? unit->weight[column] : 0.0f;
			const uint32_t bits = mx_bfloat16_bits(__fmul_rn(__fmul_rn(gated, bounded_up), weight));
			/* the block's E8M0 code, as activation_quantize_load finds it */
			const uint32_t largest = __reduce_max_sync(0xFFFFFFFFu, bits & 0x7FFFu);
			const float ratio = __fmul_rn(fmaxf(__uint_as_float(largest << 16), 1.0e-4f), 1.0f / 448.0f);
			const uint32_t ratio_bits = __float_as_uint(ratio);
			const uint32_t code = (ratio_bits >> 23) + ((ratio_bits & 0x007FFFFFu) != 0 ? 1u : 0u);
			if (lane == i + j)
				exponent = code;
			hidden[j] = __fmul_rn(__uint_as_float(bits << 16), __uint_as_float((254u - code) << 23));
			sign[j] = (bits >> 8) & 0x80u;
		}
		const uint32_t both = __nv_cvt_float2_to_fp8x2(make_float2(hidden[0], hidden[1]), __NV_SATFINITE, __NV_E4M3);
		codes[i * 32u + at] = (unsigned char)((both & 0x7Fu) | sign[0]);
		codes[(i + 1u) * 32u + at] = (unsigned char)(((both >> 8) & 0x7Fu) | sign[1]);
	}
	__syncwarp();
	/* eight rows' 32 codes and their exponents: by vector, or in the operand order of the down launch's tiles */
	const uint32_t I = arguments.output_size, column = first + lane / 2u;
	const bool routed = unit->kind == MX_UNIT_ROUTED;
	if (lane < 16u && column < unit->rows) {
		unsigned char *to;
		if (FEW)
			to = arena + (routed ? arguments.output_offset : arguments.shared_output_offset) +
			     (uint64_t)unit->vector[column] * I + unit->group * 64u + q * 32u + lane % 2u * 16u;
		else
			to = arena + arguments.output_offset + (uint64_t)unit->tile * MX_TILE_ROWS * I +
			     (unit->group * 4u + q * 2u + lane % 2u) * MX_PIECE + column * 16u;
		*reinterpret_cast<uint4 *>(to) = *reinterpret_cast<const uint4 *>(codes + lane * 16u);
	}
	if (lane < 8u && first + lane < unit->rows) {
		const uint32_t row = first + lane;
		if (FEW)
			arena[(routed ? arguments.output_exponents_offset : arguments.shared_output_exponents_offset) +
			      (uint64_t)unit->vector[row] * (I / 32u) + unit->group * 2u + q] = (unsigned char)exponent;
		else
			arena[arguments.output_exponents_offset +
			      ((uint64_t)unit->tile * (I / MX_BLOCK_INPUTS) + unit->group / 2u) * MX_SCALE_BYTES + row % 32u * 16u +
			      row / 32u * 4u + unit->group % 2u * 2u + q] = (unsigned char)exponent;
	}
	__syncwarp();
}

/* Sixteen columns of a down unit: bfloat16 outputs, two adjacent ones a store (lanes of a pair swap columns). */
__device__ __forceinline__ void mx_outputs(const struct mx_products_arguments &arguments, unsigned char *arena,
					   const struct mx_unit *unit, const float sums[16], uint32_t chunk, uint32_t lane,
					   uint32_t warp)
{
	const uint32_t odd = lane % 2u;
	unsigned char *const output =
		arena + (unit->kind == MX_UNIT_ROUTED ? arguments.output_offset : arguments.shared_output_offset) +
		(unit->group * 128u + warp % 4u * 32u + lane - odd) * 2u;
#pragma unroll
	for (uint32_t i = 0; i < 16; i += 2) {
		const uint32_t even_column = mx_bfloat16_bits(sums[i]), odd_column = mx_bfloat16_bits(sums[i + 1u]);
		const uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, odd != 0 ? even_column : odd_column, 1);
		const uint32_t column = chunk * 16u + i + odd;
		if (column < unit->rows)
			*reinterpret_cast<uint32_t *>(output + (uint64_t)unit->vector[column] * arguments.output_size * 2u) =
				odd != 0 ? other | odd_column << 16 : even_column | other << 16;
	}
}

template <bool DOWN, bool FEW>
__device__ __forceinline__ void mx_epilogue(const struct mx_products_arguments &arguments, unsigned char *arena,
					    struct mx_shared &shared, unsigned char *dynamic_shared, uint32_t lane, uint32_t warp)
{
	typedef mx_form<FEW> form;
	constexpr uint32_t sets = form::epilogue_warps / 4u; /* of four warps; a set takes every `sets`-th chunk of columns */
	const uint32_t blocks = arguments.input_size / MX_BLOCK_INPUTS;
	const uint32_t quarter = shared.tensor_memory + (warp % 4u * 32u << 16);
	struct mx_place place = { 0 };
	uint32_t count = 0, turn = 0;
	for (;;) {
		const struct mx_unit *const unit = place.peek(shared);
		if (!mx_agree<form::epilogue_warps>(unit != nullptr) || unit->kind == MX_UNIT_END)
			return;
		bool good = true;
		const uint32_t chunks = (unit->rows + 15u) / 16u;
		if (unit->kind == MX_UNIT_SHARED && arguments.shared_format == WEIGHT_FORMAT_E4M3_BLOCK128) {
			/* one FP32 scale per 128 outputs and block; a set's chunk (FEW: both chunks) of the unit's columns */
			constexpr uint32_t held = MX_BLOCK128_ROWS / 16u / sets;
			const float *const scales =
				reinterpret_cast<const float *>(unit->matrix[warp % 4u / 2u] +
								(uint64_t)arguments.output_size * arguments.input_size) +
				(uint64_t)(DOWN ? unit->group : unit->group / 2u) * blocks;
			float total[held][16];
#pragma unroll
			for (uint32_t h = 0; h < held; h++)
#pragma unroll
				for (uint32_t i = 0; i < 16; i++)
					total[h][i] = 0.0f;
			for (uint32_t block = 0; block < blocks; block++, count++) {
				const float scale = __ldg(scales + block);
				good = mx_wait(&shared.sum_full[count % 2u], (count / 2u) & 1u);
				if (!good)
					break;
				mx_fence_after();
#pragma unroll
				for (uint32_t h = 0; h < held; h++)
					if (h * sets + warp / 4u < chunks) {
						float sums[16];
						mx_load_sums(quarter + count % 2u * 128u + (h * sets + warp / 4u) * 16u, sums);
#pragma unroll
						for (uint32_t i = 0; i < 16; i++)
							total[h][i] = __fmaf_rn(sums[i], scale, total[h][i]);
					}
				mx_fence_before();
				__syncwarp();
				if (lane == 0)
					barrier_arrive(&shared.sum_free[count % 2u]);
			}
			if (!mx_agree<form::epilogue_warps>(good))
				return;
#pragma unroll
			for (uint32_t h = 0; h < held; h++)
				if (h * sets + warp / 4u < chunks) {
					if (DOWN)
						mx_outputs(arguments, arena, unit, total[h], h * sets + warp / 4u, lane, warp);
					else
						mx_hidden<FEW>(arguments, arena, unit, dynamic_shared, total[h], h * sets + warp / 4u, turn++,
							       lane, warp);
				}
		} else {
			if (!mx_agree<form::epilogue_warps>(mx_wait(&shared.sum_full[count % 2u], (count / 2u) & 1u)))
				return;
			mx_fence_after();
			for (uint32_t chunk = warp / 4u; chunk < chunks; chunk += sets) {
				float sums[16];
				mx_load_sums(quarter + count % 2u * 128u + chunk * 16u, sums);
				if (DOWN)
					mx_outputs(arguments, arena, unit, sums, chunk, lane, warp);
				else
					mx_hidden<FEW>(arguments, arena, unit, dynamic_shared, sums, chunk, turn++, lane, warp);
			}
			mx_fence_before();
			__syncwarp();
			if (lane == 0)
				barrier_arrive(&shared.sum_free[count % 2u]);
			count++;
		}
		place.release(shared, lane);
	}
}

/* ------------------------------------------------------------------ the launches */

template <bool DOWN, bool FEW>
__device__ __forceinline__ void mx_run(const struct mx_products_arguments &arguments, unsigned char *arena,
				       unsigned char *dynamic_shared, struct mx_shared &shared)
{
	typedef mx_form<FEW> form;
	/* once a wait has run out (the flag stays set while the kernel file is loaded) later CTAs do not queue up behind the
	 * same fault: the host reads the flag and rejects the result */
	if (__syncthreads_or(*reinterpret_cast<volatile unsigned int *>(&exl3_wait_expired) != 0u))
		return;
	const uint32_t lane = threadIdx.x % EXL3_WARP, warp = threadIdx.x / EXL3_WARP;
	if (threadIdx.x == 0) {
		for (uint32_t slot = 0; slot < MX_UNITS; slot++) {
			barrier_init(&shared.unit_full[slot], 1);
			/* the weights', the rows', the multiplying and the epilogue's warps */
			barrier_init(&shared.unit_free[slot],
				     MX_WEIGHT_WARPS + form::row_warps + 1u + form::epilogue_warps);
		}
		for (uint32_t stage = 0; stage < form::stages; stage++) {
			barrier_init(&shared.full[stage], form::team_warps + 1u); /* the stage's team, and the warp that brings its rows */
			barrier_init(&shared.empty[stage], 1);
		}
		for (uint32_t sum = 0; sum < 2u; sum++) {
			barrier_init(&shared.sum_full[sum], 1);
			barrier_init(&shared.sum_free[sum], form::epilogue_warps);
		}
		barrier_init(&shared.done, 1);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == form::multiply) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
				     smem_address(&shared.tensor_memory)),
			     "n"(512)
			     : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	mx_fence_before();
	__syncthreads();
	mx_fence_after();
	/* gate/up: everything read is the router's and the quantizer's. Down: the hidden vectors alone are the launch's
	 * before this one (the rows' warps wait for them); the tiles are older than that launch, which waited for them. */
	if (!DOWN)
		asm volatile("griddepcontrol.wait;" ::: "memory");
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	if (warp < form::epilogue_warps) {
		mx_epilogue<DOWN, FEW>(arguments, arena, shared, dynamic_shared, lane, warp);
	} else if (warp == form::multiply) {
		mx_products<FEW>(arguments, shared, dynamic_shared, lane);
	} else if (warp == form::schedule) {
		mx_schedule<DOWN, FEW>(arguments, arena, shared, lane);
	} else if (warp >= MX_WARP_WEIGHTS) {
		const uint32_t team = (warp - MX_WARP_WEIGHTS) / form::team_warps, tile = (warp - MX_WARP_WEIGHTS) % form::team_warps;
		struct mx_weights_place<form::stages> place = { { 0u }, { team, 0u }, 0u };
		if (mx_weights<DOWN, FEW, true>(arguments, arena, shared, dynamic_shared, lane, team, tile, place))
			(void)mx_weights<DOWN, FEW, false>(arguments, arena, shared, dynamic_shared, lane, team, tile, place);
	} else if (warp < form::rows + form::row_warps) {
		if (DOWN)
			asm volatile("griddepcontrol.wait;" ::: "memory");
		if (FEW)
			mx_rows_few<DOWN>(arguments, arena, shared, dynamic_shared, lane, warp - form::rows);
		else
			mx_rows_many(arguments, shared, dynamic_shared, lane);
	}
	/* a CTA whose wait ran out has no bulk copy in flight any more: the wait that ran out is far longer than a copy */
	mx_fence_before();
	__syncthreads();
	if (warp == form::multiply) {
		mx_fence_after();
		__syncwarp();
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(shared.tensor_memory), "n"(512)
			     : "memory");
	}
}

#define MX_ENTRY(name, down, few)                                                  \
	extern "C" __global__ void __launch_bounds__(MX_THREADS, 1)                \
		name(struct mx_products_arguments arguments, unsigned char *arena) \
	{                                                                          \
		extern __shared__ __align__(1024) unsigned char dynamic_shared[];  \
		__shared__ struct mx_shared shared;                                \
		mx_run<down, few>(arguments, arena, dynamic_shared, shared);       \
	}
MX_ENTRY(mx_gate_up_few, false, true)
MX_ENTRY(mx_down_few, true, true)
MX_ENTRY(mx_gate_up_many, false, false)
MX_ENTRY(mx_down_many, true, false)

/* grid (blocks) x 256: a warp a load of 64 values of a live row */
extern "C" __global__ void __launch_bounds__(256) mx_quantize(struct mx_quantize_arguments arguments, unsigned char *arena)
{
	const struct step_block step = *reinterpret_cast<const struct step_block *>(arena + arguments.step_offset);
	const uint32_t loads = arguments.base.width / LINEAR_VALUES_PER_LOAD;
	const uint32_t tasks = min(step.row_count, arguments.row_capacity) * loads, warps = blockDim.x / 32u;
	for (uint32_t task = blockIdx.x * warps + threadIdx.x / 32u; task < tasks; task += gridDim.x * warps)
		activation_quantize_load<true>(arguments.base, arena, task / loads, task % loads, threadIdx.x % 32u,
					       arguments.stream_offset);
}

/* grid (tiles of 128 rows, ceil(width / 512)) x 256: the rows of a tile in operand order: the sixteen bytes of row r and
 * inputs 16 c .. 16 c + 15 (in stream order) at byte 2048 c + 16 r of the tile, its scales of 128 inputs as tcgen05.cp
 * takes them. Tiles behind the routed ones are consecutive rows, the always-on expert's. A warp moves eight rows by 64
 * inputs a turn: 64 contiguous bytes a row in, 128 contiguous bytes a piece out. */
extern "C" __global__ void __launch_bounds__(256) mx_gather(struct mx_gather_arguments arguments, unsigned char *arena)
{
	const struct step_block step = *reinterpret_cast<const struct step_block *>(arena + arguments.step_offset);
	const uint32_t live = min(step.row_count, arguments.row_capacity), width = arguments.width, tile = blockIdx.x;
	const uint32_t lane = threadIdx.x % EXL3_WARP, warp = threadIdx.x / EXL3_WARP;
	const struct exl3_prefill_entry *entries = nullptr;
	uint32_t rows, base = 0;
	if (tile < arguments.tile_capacity) {
		if (tile >= reinterpret_cast<const uint32_t *>(arena + arguments.counts_offset)[arguments.expert_count])
			return;
		const struct exl3_prefill_tile record =
			reinterpret_cast<const struct exl3_prefill_tile *>(arena + arguments.tiles_offset)[tile];
		rows = record.row_count;
		entries = reinterpret_cast<const struct exl3_prefill_entry *>(arena + arguments.entries_offset) +
			  (uint64_t)record.expert * arguments.row_capacity + record.first_entry;
	} else {
		const uint32_t shared_rows = mx_shared_tile_rows(arguments.shared_format);
		base = (tile - arguments.tile_capacity) * shared_rows;
		rows = base < live ? min(live - base, shared_rows) : 0u;
	}
	unsigned char *const codes_to = arena + arguments.tile_codes_offset + (uint64_t)tile * MX_TILE_ROWS * width;
	unsigned char *const scales_to =
		arena + arguments.tile_exponents_offset + (uint64_t)tile * (width / MX_BLOCK_INPUTS) * MX_SCALE_BYTES;
	const uint32_t first = blockIdx.y * 512u, inputs = min(width - first, 512u);
	for (uint32_t row = warp * 8u + lane % 8u; row < rows; row += 64u) {
		const uint64_t source = entries != nullptr ? entries[row].pair / arguments.pairs_per_row : base + row;
		const unsigned char *const from = arena + arguments.codes_offset + source * width + first;
		for (uint32_t piece = lane / 8u; piece < inputs / 16u; piece += 4u)
			*reinterpret_cast<uint4 *>(codes_to + (uint64_t)(first / 16u + piece) * MX_PIECE + row * 16u) =
				*reinterpret_cast<const uint4 *>(from + piece * 16u);
		const uint32_t block = lane / 8u;
		if (block < inputs / MX_BLOCK_INPUTS)
			*reinterpret_cast<uint32_t *>(scales_to + (uint64_t)(first / MX_BLOCK_INPUTS + block) * MX_SCALE_BYTES +
						      row % 32u * 16u + row / 32u * 4u) =
				*reinterpret_cast<const uint32_t *>(arena + arguments.exponents_offset + source * (width / 32u) +
								    first / 32u + block * 4u);
	}
}
