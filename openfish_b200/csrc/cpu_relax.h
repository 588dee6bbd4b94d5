// cpu_relax.h -- what a host thread does between two looks at a word that the GPU will write.  Plain C++ for any host.
#pragma once

inline void cpu_relax() {
#if defined(__x86_64__) || defined(__i386__)
    __builtin_ia32_pause();
#elif defined(__aarch64__)
    asm volatile("yield");
#endif
}
