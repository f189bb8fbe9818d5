/* copy_pool.c: host memory copies by a few threads at once (copy_pool.h). */
#include "copy_pool.h"
#include "processor.h"

#include <pthread.h>
#include <sched.h>
#include <string.h>
#include <unistd.h>

#ifdef __SSE2__
#include <emmintrin.h>
#endif

#define POOL_THREADS_MOST 3u /* beside the caller: four copy 16.8 MB in 0.32 ms, eight in 0.28 */

static pthread_mutex_t mutex = PTHREAD_MUTEX_INITIALIZER;
static pthread_cond_t wake = PTHREAD_COND_INITIALIZER;
static pthread_t threads[POOL_THREADS_MOST];
static uint32_t thread_count, users;
static bool ending;
static struct ab_copy_batch *current; /* one batch at a time: another caller copies by itself */

/* Stores past the caches: what the device reads next lies in memory and not as dirty lines of some core's cache, which
 * PCIe reads at half its rate (a prompt of 2048 rows of 4096, 16.8 MB and 2 MB of scores: 1042 us, so 565). */
#ifdef __SSE2__
static void copy_past_caches(void *to, const void *from, size_t byte_count)
{
	unsigned char *out = to;
	const unsigned char *in = from;
	const size_t head = (16u - ((uintptr_t)out & 15u)) & 15u;
	if (byte_count < 64u + head) {
		memcpy(out, in, byte_count);
		return;
	}
	memcpy(out, in, head);
	out += head, in += head, byte_count -= head;
	for (; byte_count >= 64u; out += 64, in += 64, byte_count -= 64u)
		for (int quarter = 0; quarter < 4; quarter++)
			_mm_stream_si128((__m128i *)(void *)(out + 16 * quarter),
					 _mm_loadu_si128((const __m128i *)(const void *)(in + 16 * quarter)));
	_mm_sfence();
	memcpy(out, in, byte_count);
}
#else /* another processor: its own copy */
static void copy_past_caches(void *to, const void *from, size_t byte_count)
{
	memcpy(to, from, byte_count);
}
#endif

static void copy_make(struct ab_copy_batch *batch, uint32_t index)
{
	const struct ab_copy *const copy = &batch->copies[index];
	if (batch->to_device)
		copy_past_caches(copy->to, copy->from, copy->byte_count);
	else
		memcpy(copy->to, copy->from, copy->byte_count);
	__atomic_store_n(&batch->done[index], 1u, __ATOMIC_RELEASE); /* the batch may be gone after this */
}

static void *pool_thread(void *unused)
{
	(void)unused;
	(void)pthread_mutex_lock(&mutex);
	while (!ending) {
		if (current != NULL && current->soon && current->next >= current->allowed && current->next < current->count) {
			(void)pthread_mutex_unlock(&mutex);
			for (uint32_t turn = 0; turn < 32u; turn++)
				processor_pause();
			(void)pthread_mutex_lock(&mutex);
			continue;
		}
		if (current == NULL || current->next >= current->allowed) {
			(void)pthread_cond_wait(&wake, &mutex);
			continue;
		}
		struct ab_copy_batch *const batch = current;
		const uint32_t index = batch->next++;
		(void)pthread_mutex_unlock(&mutex);
		copy_make(batch, index);
		(void)pthread_mutex_lock(&mutex);
	}
	(void)pthread_mutex_unlock(&mutex);
	return NULL;
}

void ab_copy_pool_enter(void)
{
	(void)pthread_mutex_lock(&mutex);
	users++;
	(void)pthread_mutex_unlock(&mutex);
}

void ab_copy_pool_leave(void)
{
	pthread_t ended[POOL_THREADS_MOST];
	uint32_t count = 0;
	(void)pthread_mutex_lock(&mutex);
	if (--users == 0) {
		count = thread_count;
		memcpy(ended, threads, sizeof(ended));
		thread_count = 0;
		ending = count != 0;
		(void)pthread_cond_broadcast(&wake);
	}
	(void)pthread_mutex_unlock(&mutex);
	for (uint32_t thread = 0; thread < count; thread++)
		(void)pthread_join(ended[thread], NULL);
	if (count != 0) {
		(void)pthread_mutex_lock(&mutex);
		ending = false;
		(void)pthread_mutex_unlock(&mutex);
	}
}

void ab_copy_batch_begin(struct ab_copy_batch *batch)
{
	batch->next = 0;
	batch->shared = batch->soon = false;
	memset(batch->done, 0, sizeof(batch->done));
	if (batch->count < 2)
		return; /* not worth waking anyone */
	(void)pthread_mutex_lock(&mutex);
	const long cores = sysconf(_SC_NPROCESSORS_ONLN);
	while (!ending && thread_count < POOL_THREADS_MOST && (long)thread_count + 1 < cores &&
	       pthread_create(&threads[thread_count], NULL, pool_thread, NULL) == 0)
		thread_count++;
	batch->shared = current == NULL && thread_count != 0;
	if (batch->shared) {
		current = batch;
		if (batch->allowed != 0)
			(void)pthread_cond_broadcast(&wake);
	}
	(void)pthread_mutex_unlock(&mutex);
}

void ab_copy_batch_allow(struct ab_copy_batch *batch, uint32_t allowed)
{
	(void)pthread_mutex_lock(&mutex);
	batch->allowed = allowed;
	if (batch->shared)
		(void)pthread_cond_signal(&wake);
	(void)pthread_mutex_unlock(&mutex);
}

void ab_copy_batch_soon(struct ab_copy_batch *batch)
{
	(void)pthread_mutex_lock(&mutex);
	if (batch->shared && !batch->soon) {
		batch->soon = true;
		(void)pthread_cond_broadcast(&wake);
	}
	(void)pthread_mutex_unlock(&mutex);
}

void ab_copy_batch_cut(struct ab_copy_batch *batch)
{
	(void)pthread_mutex_lock(&mutex);
	batch->count = batch->allowed;
	(void)pthread_mutex_unlock(&mutex);
}

bool ab_copy_batch_help(struct ab_copy_batch *batch)
{
	(void)pthread_mutex_lock(&mutex);
	const bool taken = batch->next < batch->allowed;
	const uint32_t index = taken ? batch->next++ : 0u;
	(void)pthread_mutex_unlock(&mutex);
	if (taken)
		copy_make(batch, index);
	return taken;
}

bool ab_copy_batch_is_done(const struct ab_copy_batch *batch, uint32_t copy)
{
	return __atomic_load_n(&batch->done[copy], __ATOMIC_ACQUIRE) != 0;
}

void ab_copy_batch_end(struct ab_copy_batch *batch)
{
	ab_copy_batch_allow(batch, batch->count);
	while (ab_copy_batch_help(batch))
		;
	(void)pthread_mutex_lock(&mutex);
	if (batch->shared)
		current = NULL;
	(void)pthread_mutex_unlock(&mutex);
	for (uint32_t copy = 0; copy < batch->count; copy++)
		while (!ab_copy_batch_is_done(batch, copy))
			(void)sched_yield();
}
