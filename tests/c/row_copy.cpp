// The copies of every strip's part of every row of small frames, at every
// alignment: within the ring's slot, and never past the aligned 4-byte words that
// hold the frame's bytes.
#include <stdint.h>
#include <stdio.h>

#include <algorithm>

#include "row_copy.h"

int main() {
    const int strip = 128, step = 120;   // samples of a strip, from one strip's first to the next's
    for (int px : {3, 12})
        for (int w : {1, 2, 3, 5, 6, 11, 16, 43, 64, 127, 128, 129, 131, 250, 256})
            for (int h = 1; h <= 5; h++)
                for (int off = 0; off < 16; off += px == 12 ? 4 : 1) {
                    const uintptr_t first = 4096 + off, last = first + (uintptr_t)px * w * h;
                    for (int y = 0; y < h; y++)
                        for (int x = 0; x < w; x += step) {
                            const int x0 = x ? x - 4 : 0;
                            const int bytes = px * std::min(strip, w - x0);
                            const uintptr_t q = first + (uintptr_t)px * (y * w + x0);
                            const int unit = wema::row_inner(y, wema::inner_rows(h, px * w)) ? 16 : 4;
                            const uintptr_t a = q & ~(uintptr_t)(unit - 1), e = (q + bytes + unit - 1) & ~(uintptr_t)(unit - 1);
                            const bool ok = a >= (first & ~(uintptr_t)3) && e <= ((last + 3) & ~(uintptr_t)3) &&
                                            (int)(e - (q & ~(uintptr_t)15)) <= 16 * (strip * px / 16 + 1);
                            if (!ok) {
                                printf("px %d, %d x %d at %d: row %d from %d: units of %d\n", px, w, h, off, y, x0, unit);
                                return 1;
                            }
                        }
                }
    return 0;
}
