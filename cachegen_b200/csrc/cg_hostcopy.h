// Host memory primitives of the byte-string copies (cg_host.cu): what they need of the processor, and a portable form of
// each for any other (CG_PORTABLE_HOST selects it on x86 too).
#pragma once

#include <stdint.h>
#include <string.h>

#if defined(__x86_64__) && !defined(CG_PORTABLE_HOST)
#define CG_HOST_X86 1
#include <immintrin.h>
#else
#define CG_HOST_X86 0
#endif

namespace cg {

#if CG_HOST_X86
// Stores that bypass the cache: the bytes are not read again on this side.
__attribute__((target("avx2"))) inline void copy_streaming(uint8_t *d, const uint8_t *s, int64_t n) {
    const int64_t head = (32 - (reinterpret_cast<uintptr_t>(d) & 31)) & 31;
    if (n < 4096) {
        memcpy(d, s, static_cast<size_t>(n));
        return;
    }
    memcpy(d, s, static_cast<size_t>(head));
    d += head;
    s += head;
    n -= head;
    for (; n >= 128; n -= 128, d += 128, s += 128) {
        const __m256i a = _mm256_loadu_si256(reinterpret_cast<const __m256i *>(s));
        const __m256i b = _mm256_loadu_si256(reinterpret_cast<const __m256i *>(s + 32));
        const __m256i c = _mm256_loadu_si256(reinterpret_cast<const __m256i *>(s + 64));
        const __m256i e = _mm256_loadu_si256(reinterpret_cast<const __m256i *>(s + 96));
        _mm256_stream_si256(reinterpret_cast<__m256i *>(d), a);
        _mm256_stream_si256(reinterpret_cast<__m256i *>(d + 32), b);
        _mm256_stream_si256(reinterpret_cast<__m256i *>(d + 64), c);
        _mm256_stream_si256(reinterpret_cast<__m256i *>(d + 96), e);
    }
    memcpy(d, s, static_cast<size_t>(n));
    _mm_sfence();
}
#endif

inline void copy_piece(uint8_t *d, const uint8_t *s, int64_t n) {
#if CG_HOST_X86
    static const bool avx2 = __builtin_cpu_supports("avx2");
    if (avx2) {
        copy_streaming(d, s, n);
        return;
    }
#endif
    memcpy(d, s, static_cast<size_t>(n));
}

// Between two looks at a word that another thread writes.
inline void spin_pause() {
#if CG_HOST_X86
    _mm_pause();
#elif defined(__aarch64__)
    asm volatile("yield" ::: "memory");
#endif
}

// Makes the page present and writable; its bytes, which another thread may be writing, stay what they are.
inline void touch_page(uint8_t *p) {
#if CG_HOST_X86
    asm volatile("lock; orb $0, %0" : "+m"(*p));
#else
    __atomic_fetch_or(p, static_cast<uint8_t>(0), __ATOMIC_RELAXED);
#endif
}

}  // namespace cg
