/*
 * copy_pool.h: host memory copies by a few threads at once: a prompt's rows and results cross ordinary memory on their
 * way to and from page-locked memory, and one core moves 18 GB/s where PCIe moves 53 (16.8 MB: 0.93 ms by one thread,
 * 0.32 by four). Private to csrc/host. The threads start with the first batch and live until the last user has left.
 */
#ifndef AB_COPY_POOL_H
#define AB_COPY_POOL_H

#include <stdbool.h>
#include <stddef.h>
#include <stdint.h>

#define AB_COPY_BATCH_MOST 64u

struct ab_copy {
	void *to;
	const void *from;
	size_t byte_count;
};

/* Copies handed out in ascending order; `allowed` of them may be taken yet. done[i] is set once copy i is made. */
struct ab_copy_batch {
	struct ab_copy copies[AB_COPY_BATCH_MOST];
	uint32_t count;
	uint32_t next, allowed; /* under the pool's mutex */
	uint32_t done[AB_COPY_BATCH_MOST];
	bool to_device; /* the copies' targets are read by the device next: written past the caches */
	bool shared; /* the pool's threads help (else they are busy with another thread's batch) */
	bool soon; /* under the pool's mutex: the rest will be allowed within microseconds */
};

void ab_copy_pool_enter(void); /* one more user (a card opens) */
void ab_copy_pool_leave(void); /* the last one ends the threads */

/* offers the batch (copies, count and allowed filled in) to the pool; must be ended by the same thread */
void ab_copy_batch_begin(struct ab_copy_batch *batch);
void ab_copy_batch_allow(struct ab_copy_batch *batch, uint32_t allowed);
/* The rest of the batch will be allowed piece by piece from now on: the pool's threads are woken and look out for it
 * instead of being woken, 30 to 50 us each time, for every piece. */
void ab_copy_batch_soon(struct ab_copy_batch *batch);
void ab_copy_batch_cut(struct ab_copy_batch *batch); /* what is not allowed yet is not made */
bool ab_copy_batch_help(struct ab_copy_batch *batch); /* makes one copy; false: none may be taken */
bool ab_copy_batch_is_done(const struct ab_copy_batch *batch, uint32_t copy);
void ab_copy_batch_end(struct ab_copy_batch *batch); /* makes or awaits the rest */

#endif
