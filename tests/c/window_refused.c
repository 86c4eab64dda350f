/* temporal_filter_apply on a buffer whose window size temporal_buffer_init refused:
 * zeros, as before a window is full; no division by the size, no ring to read. */
#include <stdio.h>
#include <string.h>

#include "dwt.h"
#include "temporal_filter.h"

int main(void) {
    static const int sizes[] = {0, -5};
    for (int k = 0; k < 2; k++) {
        for (int bilateral = 0; bilateral < 2; bilateral++) {
            DWTCoeffs c;
            TemporalFilter f;
            TemporalBuffer b;
            float out[6 * 8 * 8];
            if (dwt_init(&c, 16, 16, 1)) return 2;
            if (temporal_filter_init(&f, 0.1f, 0.2f, 8)) return 3;
            if (temporal_buffer_init(&b, &c, sizes[k]) != -1) return 4;
            if (b.num_positions != 6 * 8 * 8) return 5;
            memset(out, 0x55, sizeof out);
            temporal_filter_apply(&f, &b, out, bilateral != 0);
            for (int i = 0; i < 6 * 8 * 8; i++)
                if (out[i] != 0.0f) { printf("size %d: [%d] = %g\n", sizes[k], i, out[i]); return 1; }
            temporal_buffer_free(&b);
            temporal_filter_free(&f);
            dwt_free(&c);
        }
    }
    return 0;
}
