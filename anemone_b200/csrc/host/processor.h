/* processor.h: what the host code asks of a processor by name, with a plain form for any other. Private to csrc/host. */
#ifndef AB_PROCESSOR_H
#define AB_PROCESSOR_H

/* between two looks at a word another thread or the device is about to write */
static inline void processor_pause(void)
{
#if defined(__x86_64__) || defined(__i386__)
	__builtin_ia32_pause();
#elif defined(__aarch64__)
	__asm__ volatile("yield" ::: "memory");
#else
	__asm__ volatile("" ::: "memory");
#endif
}

#endif
