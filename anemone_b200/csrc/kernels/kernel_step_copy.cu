/*
 * kernel_step_copy.cu: the copies of a step's own graph (backend_b200_step_capture) as kernels: a step's inputs from
 * page-locked host memory into the arena, its outputs back, and a word in host memory that says so. A few dozen
 * kilobytes: what bounds them is latency, one trip over PCIe each (about 2 us in, the stores out are posted). As memcpy
 * nodes the two copies of a decode step of eight rows added 24 us to a step of 115 us on this card (the nodes' own
 * dispatch on a copy engine and the dependencies between engines); as kernels that overlap their neighbours' launches
 * they add 7. A host that polls the word instead of the stream sees the end about 5 us earlier.
 * A range is copied in 16-byte pieces, the last bytes one by one.
 */
#include <stdint.h>

#include "anemone_b200_backend.h"

/* host memory is read past every cache: another run of the graph left other bytes there */
__device__ __forceinline__ uint4 load_host(const uint4 *address)
{
	uint4 value;
	asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
		     : "=r"(value.x), "=r"(value.y), "=r"(value.z), "=r"(value.w)
		     : "l"(address)
		     : "memory");
	return value;
}

/* a warp: the bits of up to 32 of these words (device addresses, 0: none) or-ed */
__device__ __forceinline__ unsigned int wait_bits(const uint64_t *words, uint32_t count)
{
	const uint64_t word = threadIdx.x < count ? words[threadIdx.x] : 0u;
	return __reduce_or_sync(0xFFFFFFFFu, word != 0 ? *reinterpret_cast<const volatile unsigned int *>(word) : 0u);
}

/* grid (blocks) x BACKEND_B200_STEP_COPY_THREADS */
extern "C" __global__ void __launch_bounds__(BACKEND_B200_STEP_COPY_THREADS)
	step_copy_in(struct backend_b200_step_copy_record record, unsigned char *arena)
{
	/* the step's first launch may take its place meanwhile; it waits for this one before it reads */
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	const unsigned char *const from = reinterpret_cast<const unsigned char *>(record.host_address);
	unsigned char *const to = arena + record.arena_offset;
	const uint64_t pieces = record.byte_count / 16u;
	for (uint64_t index = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; index < pieces; index += (uint64_t)gridDim.x * blockDim.x)
		reinterpret_cast<uint4 *>(to)[index] = load_host(reinterpret_cast<const uint4 *>(from) + index);
	if (blockIdx.x == 0 && threadIdx.x < record.byte_count % 16u)
		to[pieces * 16u + threadIdx.x] =
			*reinterpret_cast<const volatile unsigned char *>(from + pieces * 16u + threadIdx.x);
}

__device__ unsigned int step_copy_arrived; /* blocks of the launch that have stored their part; zero between launches */
__device__ uint64_t step_copy_runs[BACKEND_MAXIMUM_GRAPHS]; /* of a graph: the number of its last run that is done */

extern "C" __global__ void __launch_bounds__(BACKEND_B200_STEP_COPY_THREADS)
	step_copy_out(const __grid_constant__ struct backend_b200_step_copy_record record, unsigned char *arena)
{
	/* this run's number: the runs of a graph follow one another on the card's stream, and the host counts them as it
	 * queues them. (A number the host wrote before each launch would be read by every run still queued.) */
	uint64_t run = 0;
	if (threadIdx.x == 0)
		run = *reinterpret_cast<volatile uint64_t *>(&step_copy_runs[record.graph]) + 1u;
	asm volatile("griddepcontrol.wait;" ::: "memory");
	/* whether a kernel of the graph's files gave up a bounded wait: beside the copy, a word is an L2 read */
	if (blockIdx.x == 0 && threadIdx.x < 32u) {
		const unsigned int bits = wait_bits(record.wait_words, BACKEND_B200_STEP_COPY_WAIT_WORDS);
		if (threadIdx.x == 0 && bits != 0)
			*reinterpret_cast<volatile uint64_t *>(record.expired_address) = bits;
	}
	unsigned char *const to = reinterpret_cast<unsigned char *>(record.host_address);
	const unsigned char *const from = arena + record.arena_offset;
	const uint64_t pieces = record.byte_count / 16u;
	for (uint64_t index = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; index < pieces; index += (uint64_t)gridDim.x * blockDim.x)
		reinterpret_cast<uint4 *>(to)[index] = __ldcg(reinterpret_cast<const uint4 *>(from) + index);
	if (blockIdx.x == 0 && threadIdx.x < record.byte_count % 16u)
		to[pieces * 16u + threadIdx.x] = from[pieces * 16u + threadIdx.x];
	/* a fence of the device's scope a block, one of the system's scope a launch, which is cumulative over what the last
	 * block has seen counted: system fences of many blocks stand in line, 1 us each (17 us for 64 KB) */
	__syncthreads();
	if (threadIdx.x == 0) {
		__threadfence();
		if (atomicAdd(&step_copy_arrived, 1u) == gridDim.x - 1u) {
			step_copy_arrived = 0u;
			step_copy_runs[record.graph] = run;
			__threadfence_system();
			*reinterpret_cast<volatile uint64_t *>(record.done_address) = run;
		}
	}
}

/* grid (1) x 32: behind a graph, for the calls whose outputs go by memcpy */
extern "C" __global__ void __launch_bounds__(32)
	step_wait_words(const __grid_constant__ struct backend_b200_wait_words_record record, unsigned char *arena)
{
	(void)arena;
	const unsigned int bits = wait_bits(record.wait_words, BACKEND_B200_WAIT_WORDS_MOST);
	if (threadIdx.x == 0 && bits != 0)
		*reinterpret_cast<volatile uint64_t *>(record.host_address) = bits;
}
