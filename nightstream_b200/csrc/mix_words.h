// mix_words.h -- four columns of a digit row that begins on any byte, from aligned words
// (rlc_tc.cu).  Plain C++: the CPU test runs it over buffers of the exact size.
#pragma once
#include <cstdint>
#include "gl.cuh"

#ifndef NEO_D
#define NEO_D 54
#endif

// Digits of `count` witnesses of NEO_D rows of m bytes: Z[0 .. bytes).
struct MixRows {
    const int8_t* Z;
    uint64_t m, bytes;
    uint32_t count;
};

// The aligned word at address w.  A word that the buffer covers in part (its last one, when
// the digits do not end on four bytes; its first one, should they not begin there) is put
// together from the bytes inside, the others zero.
GL_HD uint32_t mix_word(const MixRows& a, uintptr_t w) {
    const uintptr_t lo = reinterpret_cast<uintptr_t>(a.Z), hi = lo + a.bytes;
    if (w >= lo && w + 4 <= hi) {
#ifdef __CUDA_ARCH__
        return __ldg(reinterpret_cast<const uint32_t*>(w));
#else
        return *reinterpret_cast<const uint32_t*>(w);
#endif
    }
    uint32_t x = 0;
    for (uint32_t b = 0; b < 4; b++)
        if (w + b >= lo && w + b < hi) x |= (uint32_t) * reinterpret_cast<const uint8_t*>(w + b) << (8 * b);
    return x;
}

// The words z, zn that hold columns c .. c + 3 of row k of witness wi (zn only where the row
// reaches into it; columns past the row's end are not stored).  Branch-free for all words but
// the buffer's last, so that a thread's loads are in flight together.
GL_HD void mix_fetch(const MixRows& a, uint32_t wi, uint32_t k, uint64_t c, uint32_t& z, uint32_t& zn) {
    const bool in = wi < a.count && c < a.m && k < NEO_D;
    const uintptr_t p = reinterpret_cast<uintptr_t>(a.Z) + (in ? ((uint64_t)wi * NEO_D + k) * a.m + c : 0);
    const uint32_t off = (uint32_t)(p & 3);
    z = mix_word(a, p - off);
    zn = mix_word(a, p - off + (in && off && c + 4 - off < a.m ? 4 : 0));
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
