// Text as a caller holds it -> UTF-8 bytes in a staging buffer.
//
// A Python string keeps its characters in one, two or four bytes each; asking the interpreter for its
// UTF-8 form makes a copy at about 1 GB/s (300 KB of mixed scripts: 0.30 ms, more than the GPU needs for
// them) that then has to be copied once more into page-locked memory.  The functions here write the UTF-8
// form straight to where the device fetches it from.
#pragma once
#include <cstddef>
#include <cstdint>

namespace gtok {

// A run of text in the caller's memory.
struct TextPiece {
    const void* data;
    uint64_t units;        // bytes (kind 1), or characters
    uint32_t kind;         // 1 bytes, copied as they are; 2 / 4 characters of that many bytes; 3 characters of one byte (U+0000..U+00FF)
};

// UTF-8 length of `units` characters of the given kind, or ~0 when one of them is a surrogate
// (which has no UTF-8 form).
uint64_t utf8_size(const void* data, uint64_t units, uint32_t kind);
// Writes the UTF-8 form to `dst` and returns the end; no byte is written past it.  The characters have
// been through utf8_size: no surrogates.
uint8_t* utf8_write(uint8_t* dst, const void* data, uint64_t units, uint32_t kind);
// The same past the caches, for text that the device fetches next: a transfer that finds its lines modified
// in the cores' caches runs at half its rate (4.5 MB staged by four threads and sent: 183 us with ordinary
// stores, 117 with these).  The stores are complete when the call returns.
uint8_t* utf8_stream(uint8_t* dst, const void* data, uint64_t units, uint32_t kind);

}  // namespace gtok
