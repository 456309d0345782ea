// payload_row_fits against 128-bit arithmetic: keys around the last row that
// fits and around 2^64, row widths of 1 to 128 slots, payloads from none on.
#include <stdint.h>
#include <stdio.h>

#include <initializer_list>

#include "../../ltpmg_gb300/csrc/ltp_bounds.h"

int main() {
    const uint64_t top = ~0ull;
    for (uint64_t len : std::initializer_list<uint64_t>{0, 1, 2, 3, 127, 128, 129, 4096, (1ull << 32) - 1})
        for (uint64_t slots : std::initializer_list<uint64_t>{1, 2, 3, 64, 128})
            for (uint64_t d = 0; d < 300; d++)
                for (uint64_t key : std::initializer_list<uint64_t>{d, len - slots + d, len - slots - d, len + d,
                                                                    (1ull << 32) - d, (1ull << 32) + d, top - d}) {
                    const bool want = (unsigned __int128)key + slots <= len;
                    if (ltp::payload_row_fits(key, slots, len) != want) {
                        printf("key %llu slots %llu len %llu\n", (unsigned long long)key, (unsigned long long)slots,
                               (unsigned long long)len);
                        return 1;
                    }
                }
    puts("ok");
    return 0;
}
