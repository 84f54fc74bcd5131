// Every load of the ragged RLC mix over digit buffers as the callers allocate them (run under the
// address sanitizer), and the columns it makes of them.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include "../../nightstream_b200/csrc/mix_words.h"

int main() {
    for (uint64_t m : {1, 2, 3, 5, 6, 7, 9, 127, 129, 130, 131})
        for (uint32_t count : {1u, 2u, 3u})
            {
                const uint64_t bytes = (uint64_t)count * NEO_D * m + MIX_PAD;
                int8_t* Z = static_cast<int8_t*>(malloc(bytes));
                for (uint64_t i = 0; i < bytes; i++) Z[i] = (int8_t)(i * 37 + 11);
                const MixRows a = {Z, m, count};
                // the kernel's range: whole blocks of 128 columns, pairs of witnesses, 64 rows each
                for (uint32_t w = 0; w < (count + 1) / 2 * 2; w++)
                    for (uint32_t k = 0; k < 64; k++)
                        for (uint64_t c = 0; c < (m + 127) / 128 * 128; c += 4) {
                            uint32_t z, zn;
                            mix_fetch(a, w, k, c, z, zn);
                            const uint32_t q = mix_quad(a, w, k, c, z, zn);
                            for (uint32_t b = 0; b < 4 && c + b < m; b++) {
                                const int8_t want = w < count && k < NEO_D ? Z[((uint64_t)w * NEO_D + k) * m + c + b] : 0;
                                if ((int8_t)(q >> (8 * b)) != want) {
                                    printf("m %llu count %u: witness %u row %u column %llu\n", (unsigned long long)m,
                                           count, w, k, (unsigned long long)(c + b));
                                    return 1;
                                }
                            }
                        }
                free(Z);
            }
    puts("ok");
    return 0;
}
