// A hint to the host CPU that a short wait is on, for the hosts B200s come with.
#pragma once

static inline void hs_pause() {
#if defined(__x86_64__) || defined(__i386__)
  __builtin_ia32_pause();
#elif defined(__aarch64__)
  __asm__ __volatile__("yield" ::: "memory");
#endif
}
