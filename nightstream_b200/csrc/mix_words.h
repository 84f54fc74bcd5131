// mix_words.h -- four columns of a digit row that begins on any byte, from aligned words
// (rlc_tc.cu).  Plain C++: the CPU test runs it over such buffers.
#pragma once
#include <cstdint>
#include "gl.cuh"

#ifndef NEO_D
#define NEO_D 54
#endif

// Digits of `count` witnesses of NEO_D rows of m bytes at Z, which begins on four bytes and is
// followed by MIX_PAD readable bytes, so that the word of the last columns is inside the buffer
// (guarded words, put together from bytes at the buffer's end, made 13 witnesses of 2^14 - 1
// columns 27 us instead of 15).
constexpr uint64_t MIX_PAD = 3;
struct MixRows {
    const int8_t* Z;
    uint64_t m;
    uint32_t count;
};

GL_HD uint32_t mix_word(uintptr_t w) {
#ifdef __CUDA_ARCH__
    return __ldg(reinterpret_cast<const uint32_t*>(w));
#else
    return *reinterpret_cast<const uint32_t*>(w);
#endif
}

// The words z, zn that hold columns c .. c + 3 of row k of witness wi (zn only where the row
// reaches into it; columns past the row's end are not stored).  Branch-free, so that a thread's
// loads are in flight together.
GL_HD void mix_fetch(const MixRows& a, uint32_t wi, uint32_t k, uint64_t c, uint32_t& z, uint32_t& zn) {
    const bool in = wi < a.count && c < a.m && k < NEO_D;
    const uintptr_t p = reinterpret_cast<uintptr_t>(a.Z) + (in ? ((uint64_t)wi * NEO_D + k) * a.m + c : 0);
    const uint32_t off = (uint32_t)(p & 3);
    z = mix_word(p - off);
    zn = mix_word(p - off + (in && off && c + 4 - off < a.m ? 4 : 0));
}
// the four columns as one word (byte b: column c + b); zero for a row that is not there
GL_HD uint32_t mix_quad(const MixRows& a, uint32_t wi, uint32_t k, uint64_t c, uint32_t z, uint32_t zn) {
    if (wi >= a.count || c >= a.m || k >= NEO_D) return 0;
    const uintptr_t p = reinterpret_cast<uintptr_t>(a.Z) + ((uint64_t)wi * NEO_D + k) * a.m + c;
#ifdef __CUDA_ARCH__
    return __funnelshift_r(z, zn, 8 * (uint32_t)(p & 3));
#else
    return (uint32_t)((((uint64_t)zn << 32) | z) >> (8 * (p & 3)));
#endif
}
