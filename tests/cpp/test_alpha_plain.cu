// make_books_plain of tx_device.cuh, run on the host for every range of values
// that takes it, against make_book5 and make_book7 after fix_range.
#include "tx_device.cuh"

#include <cstdio>

static bool differ(const tx::AlphaBook &a, const tx::AlphaBook &b) {
    for (int j = 0; j < 7; ++j)
        if (a.t[j] != b.t[j]) return true;
    return a.idx_lo != b.idx_lo || a.idx_hi != b.idx_hi || a.val_lo != b.val_lo || a.val_hi != b.val_hi;
}

int main() {
    long ranges = 0, bad = 0;
    for (int lo = 1; lo < 255; ++lo)
        for (int hi = lo; hi < 255; ++hi) {
            if (lo > 248 && hi - lo < 7) continue;  // takes the general books
            ++ranges;
            int min5 = lo, max5 = hi, min7 = lo, max7 = hi;
            tx::fix_range(min5, max5, 5);
            tx::fix_range(min7, max7, 7);
            uint32_t c5[8] = {(uint32_t)min5, (uint32_t)max5}, c7[8] = {(uint32_t)min5, (uint32_t)max5};
            for (int i = 1; i < 5; ++i) c5[1 + i] = (uint32_t)(((5 - i) * min5 + i * max5) / 5);
            c5[6] = 0;
            c5[7] = 255;
            for (int i = 1; i < 7; ++i) c7[1 + i] = (uint32_t)(((7 - i) * min7 + i * max7) / 7);
            tx::AlphaBook a, b;
            tx::make_books_plain((uint32_t)lo, (uint32_t)(hi > lo + 5 ? hi : lo + 5), (uint32_t)(hi > lo + 7 ? hi : lo + 7), a, b);
            if (differ(a, tx::make_book5((uint32_t)min5, (uint32_t)max5, c5)) ||
                differ(b, tx::make_book7((uint32_t)min5, (uint32_t)max5, c7))) {
                if (++bad < 5) std::printf("range %d .. %d\n", lo, hi);
            }
        }
    std::printf("%ld ranges, %ld differ\n", ranges, bad);
    return bad != 0;
}
