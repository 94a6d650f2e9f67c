// Host copies into page-locked staging buffers that the copy engine reads next.
#pragma once

#include <string.h>

#include <cstddef>
#include <cstdint>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

namespace dlb {

// Copies of this size and more bypass the caches.
constexpr size_t STREAM_COPY_BYTES = (size_t)256 << 10;

// dst and src need not be aligned.  streaming: the bytes are written past the
// caches (non-temporal stores), so that the copy engine finds them in memory:
// it reads freshly written cache lines of several cores at 17 - 30 GB/s, memory
// at 54 (32 MB gathered by 4 - 16 threads on a B200 host), and the copy itself
// need not fetch the lines it overwrites (8 threads: 78 GB/s instead of 61).
// staging_fence ends a series of copies: a DMA started behind it sees the bytes.
inline void staging_copy(void *dst, const void *src, size_t bytes, bool streaming) {
#if defined(__SSE2__)
  if (streaming) {
    char *d = static_cast<char *>(dst);
    const char *s = static_cast<const char *>(src);
    const size_t head = (16 - (reinterpret_cast<uintptr_t>(d) & 15)) & 15;
    if (head < bytes) {
      memcpy(d, s, head);
      size_t i = head;
      for (; i + 64 <= bytes; i += 64) {
        const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i *>(s + i));
        const __m128i b = _mm_loadu_si128(reinterpret_cast<const __m128i *>(s + i + 16));
        const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i *>(s + i + 32));
        const __m128i e = _mm_loadu_si128(reinterpret_cast<const __m128i *>(s + i + 48));
        _mm_stream_si128(reinterpret_cast<__m128i *>(d + i), a);
        _mm_stream_si128(reinterpret_cast<__m128i *>(d + i + 16), b);
        _mm_stream_si128(reinterpret_cast<__m128i *>(d + i + 32), c);
        _mm_stream_si128(reinterpret_cast<__m128i *>(d + i + 48), e);
      }
      memcpy(d + i, s + i, bytes - i);
      return;
    }
  }
#endif
  memcpy(dst, src, bytes);
}
inline void staging_fence(bool streaming) {
#if defined(__SSE2__)
  if (streaming) _mm_sfence();
#endif
}

}  // namespace dlb
