// See host_text.h.
#include "host_text.h"

#include <algorithm>
#include <cstring>

#if defined(__x86_64__)
#include <immintrin.h>
#define GTOK_X86 1
#endif

namespace gtok {

namespace {

constexpr uint64_t kBad = ~0ull;

template <class C>
uint64_t size_plain(const C* s, uint64_t n) {
    uint64_t two = 0, three = 0, four = 0, bad = 0;
    for (uint64_t i = 0; i < n; ++i) {
        const uint32_t c = s[i];
        two += c >= 0x80u;
        if (sizeof(C) > 1) {
            three += c >= 0x800u;
            bad += (c & 0xFFFFF800u) == 0xD800u;
        }
        if (sizeof(C) > 2) four += c >= 0x10000u;
    }
    return bad ? kBad : n + two + three + four;
}

template <class C>
uint8_t* write_plain(uint8_t* d, const C* s, uint64_t n) {
    for (uint64_t i = 0; i < n; ++i) {
        const uint32_t c = s[i];
        if (c < 0x80u) { *d++ = static_cast<uint8_t>(c); continue; }
        if (c < 0x800u) {
            d[0] = static_cast<uint8_t>(0xC0u | (c >> 6));
            d[1] = static_cast<uint8_t>(0x80u | (c & 63u));
            d += 2;
        } else if (c < 0x10000u) {
            d[0] = static_cast<uint8_t>(0xE0u | (c >> 12));
            d[1] = static_cast<uint8_t>(0x80u | ((c >> 6) & 63u));
            d[2] = static_cast<uint8_t>(0x80u | (c & 63u));
            d += 3;
        } else {
            d[0] = static_cast<uint8_t>(0xF0u | (c >> 18));
            d[1] = static_cast<uint8_t>(0x80u | ((c >> 12) & 63u));
            d[2] = static_cast<uint8_t>(0x80u | ((c >> 6) & 63u));
            d[3] = static_cast<uint8_t>(0x80u | (c & 63u));
            d += 4;
        }
    }
    return d;
}

#if GTOK_X86
// Sixteen characters a step: each spread over the four bytes of a 32-bit lane with its UTF-8 bytes from
// the lowest up, the bytes that a shorter form does not have squeezed out (vpcompressb).
__attribute__((target("avx512f,avx512bw,avx512vbmi2"))) inline __m512i lanes_of(__m512i c, __mmask64* keep) {
    const __m512i k3f = _mm512_set1_epi32(0x3F), k80 = _mm512_set1_epi32(0x80);
    const __mmask16 m2 = _mm512_cmpge_epu32_mask(c, k80), m3 = _mm512_cmpge_epu32_mask(c, _mm512_set1_epi32(0x800)),
                    m4 = _mm512_cmpge_epu32_mask(c, _mm512_set1_epi32(0x10000));
    const __m512i last = _mm512_or_si512(_mm512_and_si512(c, k3f), k80);
    const __m512i mid = _mm512_or_si512(_mm512_and_si512(_mm512_srli_epi32(c, 6), k3f), k80);
    __m512i w = c;
    // two bytes: 110xxxxx 10xxxxxx
    w = _mm512_mask_or_epi32(w, m2, _mm512_or_si512(_mm512_srli_epi32(c, 6), _mm512_set1_epi32(0xC0)), _mm512_slli_epi32(last, 8));
    // three: 1110xxxx 10xxxxxx 10xxxxxx
    const __m512i tail3 = _mm512_or_si512(_mm512_slli_epi32(mid, 8), _mm512_slli_epi32(last, 16));
    w = _mm512_mask_or_epi32(w, m3, _mm512_or_si512(_mm512_srli_epi32(c, 12), _mm512_set1_epi32(0xE0)), tail3);
    if (m4) {
        const __m512i mid4 = _mm512_or_si512(_mm512_and_si512(_mm512_srli_epi32(c, 12), k3f), k80);
        const __m512i head = _mm512_or_si512(_mm512_or_si512(_mm512_srli_epi32(c, 18), _mm512_set1_epi32(0xF0)), _mm512_slli_epi32(mid4, 8));
        w = _mm512_mask_or_epi32(w, m4, head, _mm512_or_si512(_mm512_slli_epi32(mid, 16), _mm512_slli_epi32(last, 24)));
    }
    // (no byte of a character but a whole NUL is zero, and a NUL's lane keeps its lowest byte)
    *keep = _mm512_test_epi8_mask(w, w) | 0x1111111111111111ull;
    return w;
}
template <class C>
__attribute__((target("avx512f,avx512bw,avx512vl,avx512vbmi2"))) uint8_t* write_wide(uint8_t* d, const C* s, uint64_t n) {
    uint64_t i = 0;
    for (; i + 16 <= n; i += 16) {
        __m512i c;
        if (sizeof(C) == 1) {
            const __m128i v = _mm_loadu_si128(reinterpret_cast<const __m128i*>(s + i));
            if (!_mm_movemask_epi8(v)) { _mm_storeu_si128(reinterpret_cast<__m128i*>(d), v); d += 16; continue; }
            c = _mm512_cvtepu8_epi32(v);
        } else if (sizeof(C) == 2) {
            const __m256i v = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(s + i));
            if (!_mm256_test_epi16_mask(v, _mm256_set1_epi16(static_cast<short>(0xFF80)))) {
                _mm_storeu_si128(reinterpret_cast<__m128i*>(d), _mm256_cvtepi16_epi8(v));
                d += 16;
                continue;
            }
            c = _mm512_cvtepu16_epi32(v);
        } else {
            c = _mm512_loadu_si512(s + i);
        }
        __mmask64 keep;
        const __m512i w = lanes_of(c, &keep);
        const __m512i packed = _mm512_maskz_compress_epi8(keep, w);
        const int len = __builtin_popcountll(keep);
        // whole 64 bytes while that many characters (so at least that many bytes) are still to come, else just the bytes there are
        if (n - i >= 64) _mm512_storeu_si512(d, packed);
        else _mm512_mask_storeu_epi8(d, len == 64 ? ~0ull : (1ull << len) - 1ull, packed);
        d += len;
    }
    return write_plain(d, s + i, n - i);
}
bool have_wide() {
    static const bool yes = __builtin_cpu_supports("avx512f") && __builtin_cpu_supports("avx512bw") && __builtin_cpu_supports("avx512vl") &&
                            __builtin_cpu_supports("avx512vbmi2");
    return yes;
}
// Sixty-four bytes of characters a step, the characters of each length counted from comparison masks.
__attribute__((target("avx512f,avx512bw,avx512vl,avx512vbmi2,popcnt"))) uint64_t size_wide(const uint8_t* s, uint64_t n) {
    uint64_t more = 0, i = 0;
    for (; i + 64 <= n; i += 64) more += static_cast<uint64_t>(__builtin_popcountll(_mm512_movepi8_mask(_mm512_loadu_si512(s + i))));
    return i + more + size_plain(s + i, n - i);
}
__attribute__((target("avx512f,avx512bw,avx512vl,avx512vbmi2,popcnt"))) uint64_t size_wide(const uint16_t* s, uint64_t n) {
    const __m512i k80 = _mm512_set1_epi16(0x80), k800 = _mm512_set1_epi16(0x800), kf8 = _mm512_set1_epi16(static_cast<short>(0xF800)),
                  kd8 = _mm512_set1_epi16(static_cast<short>(0xD800));
    uint64_t more = 0, i = 0;
    __mmask32 bad = 0;
    for (; i + 32 <= n; i += 32) {
        const __m512i v = _mm512_loadu_si512(s + i);
        const __mmask32 m2 = _mm512_cmpge_epu16_mask(v, k80), m3 = _mm512_cmpge_epu16_mask(v, k800);
        more += static_cast<uint64_t>(__builtin_popcountll((static_cast<uint64_t>(m2) << 32) | m3));
        bad |= _mm512_cmpeq_epi16_mask(_mm512_and_si512(v, kf8), kd8);
    }
    const uint64_t rest = size_plain(s + i, n - i);
    return bad || rest == kBad ? kBad : i + more + rest;
}
__attribute__((target("avx512f,avx512bw,avx512vl,avx512vbmi2,popcnt"))) uint64_t size_wide(const uint32_t* s, uint64_t n) {
    const __m512i k80 = _mm512_set1_epi32(0x80), k800 = _mm512_set1_epi32(0x800), k10000 = _mm512_set1_epi32(0x10000),
                  kf8 = _mm512_set1_epi32(static_cast<int>(0xFFFFF800u)), kd8 = _mm512_set1_epi32(0xD800);
    uint64_t more = 0, i = 0;
    __mmask16 bad = 0;
    for (; i + 16 <= n; i += 16) {
        const __m512i v = _mm512_loadu_si512(s + i);
        const uint64_t m2 = _mm512_cmpge_epu32_mask(v, k80), m3 = _mm512_cmpge_epu32_mask(v, k800), m4 = _mm512_cmpge_epu32_mask(v, k10000);
        more += static_cast<uint64_t>(__builtin_popcountll(m2 | (m3 << 16) | (m4 << 32)));
        bad |= _mm512_cmpeq_epi32_mask(_mm512_and_si512(v, kf8), kd8);
    }
    const uint64_t rest = size_plain(s + i, n - i);
    return bad || rest == kBad ? kBad : i + more + rest;
}
#endif

template <class C>
uint64_t size_of(const C* s, uint64_t n) {
#if GTOK_X86
    if (n >= 64 && have_wide()) return size_wide(s, n);
#endif
    return size_plain(s, n);
}
template <class C>
uint8_t* write_of(uint8_t* d, const C* s, uint64_t n) {
#if GTOK_X86
    if (n >= 32 && have_wide()) return write_wide(d, s, n);
#endif
    return write_plain(d, s, n);
}

#if GTOK_X86
// Bytes from `s` to whole 64-byte lines from `d` on (d is a line's start) by streaming stores.
__attribute__((target("avx512f"))) void stream_lines_wide(uint8_t* d, const uint8_t* s, uint64_t lines) {
    for (; lines >= 4; lines -= 4, d += 256, s += 256) {
        const __m512i a = _mm512_loadu_si512(s), b = _mm512_loadu_si512(s + 64), c = _mm512_loadu_si512(s + 128), e = _mm512_loadu_si512(s + 192);
        _mm512_stream_si512(reinterpret_cast<__m512i*>(d), a);
        _mm512_stream_si512(reinterpret_cast<__m512i*>(d + 64), b);
        _mm512_stream_si512(reinterpret_cast<__m512i*>(d + 128), c);
        _mm512_stream_si512(reinterpret_cast<__m512i*>(d + 192), e);
    }
    for (; lines; --lines, d += 64, s += 64) _mm512_stream_si512(reinterpret_cast<__m512i*>(d), _mm512_loadu_si512(s));
}
void stream_lines_plain(uint8_t* d, const uint8_t* s, uint64_t lines) {
    for (; lines; --lines, d += 64, s += 64)
        for (int k = 0; k < 64; k += 16)
            _mm_stream_si128(reinterpret_cast<__m128i*>(d + k), _mm_loadu_si128(reinterpret_cast<const __m128i*>(s + k)));
}
void stream_lines(uint8_t* d, const uint8_t* s, uint64_t lines) {
    if (have_wide()) stream_lines_wide(d, s, lines); else stream_lines_plain(d, s, lines);
}
#endif

}  // namespace

uint8_t* utf8_stream(uint8_t* dst, const void* data, uint64_t units, uint32_t kind) {
#if GTOK_X86
    if (kind == 1) {
        const uint8_t* s = static_cast<const uint8_t*>(data);
        const uint64_t head = std::min<uint64_t>(units, (64 - (reinterpret_cast<uintptr_t>(dst) & 63)) & 63), lines = (units - head) / 64;
        std::memcpy(dst, s, head);
        stream_lines(dst + head, s + head, lines);
        const uint64_t at = head + lines * 64;
        std::memcpy(dst + at, s + at, units - at);
        _mm_sfence();
        return dst + units;
    }
    // Characters go through a buffer that stays in the nearest cache; it begins as far into a line as the destination does.
    constexpr uint64_t kStep = 1024;
    const uint64_t width = kind == 3 ? 1 : kind;
    alignas(64) uint8_t buf[64 + 4 * kStep + 64];
    uint64_t held = reinterpret_cast<uintptr_t>(dst) & 63, first = held;      // bytes [first, held) of the buffer are this call's
    uint8_t* line = dst - held;                                               // where the buffer's first byte goes
    for (uint64_t i = 0; i < units; i += kStep) {
        held = static_cast<uint64_t>(utf8_write(buf + held, static_cast<const uint8_t*>(data) + i * width, std::min(kStep, units - i), kind) - buf);
        uint64_t lines = held / 64;
        if (!lines) continue;
        uint64_t done = 0;
        if (first) {                                                          // the line that this call does not begin
            std::memcpy(line + first, buf + first, 64 - first);
            first = 0;
            done = 1;
        }
        stream_lines(line + done * 64, buf + done * 64, lines - done);
        std::memcpy(buf, buf + lines * 64, 64);
        line += lines * 64;
        held -= lines * 64;
    }
    std::memcpy(line + first, buf + first, held - first);
    _mm_sfence();
    return line + held;
#else
    return utf8_write(dst, data, units, kind);
#endif
}

uint64_t utf8_size(const void* data, uint64_t units, uint32_t kind) {
    switch (kind) {
        case 2: return size_of(static_cast<const uint16_t*>(data), units);
        case 3: return size_of(static_cast<const uint8_t*>(data), units);
        case 4: return size_of(static_cast<const uint32_t*>(data), units);
        default: return units;
    }
}

uint8_t* utf8_write(uint8_t* dst, const void* data, uint64_t units, uint32_t kind) {
    switch (kind) {
        case 2: return write_of(dst, static_cast<const uint16_t*>(data), units);
        case 3: return write_of(dst, static_cast<const uint8_t*>(data), units);
        case 4: return write_of(dst, static_cast<const uint32_t*>(data), units);
        default: std::memcpy(dst, data, units); return dst + units;
    }
}

}  // namespace gtok
