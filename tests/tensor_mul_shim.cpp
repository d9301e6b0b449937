// Host build of the tensor-core product (tensor_mul.cuh): the matrix product is
// made with integers, the rest is the code that the device runs.
#include "../vkzg_b200/csrc/tensor_mul.cuh"

#include <string.h>

using namespace vkzg;

static uint64_t largest;

extern "C" {
// row i of the matrix
void shim_tm_row(int i, uint8_t *row) {
    static const TmMatrix m = tm_matrix();
    memcpy(row, m.b[i], kTmCols);
}
// r = a b / R mod p (not reduced below p); sqr: a^2
void shim_tm_mul(const uint32_t *a, const uint32_t *b, int sqr, uint32_t *r) {
    static const TmImage im = tm_image();
    const TmPart x = tm_part(a), y = tm_part(b);
    uint32_t z[kTmWords], w[kTmCols / 2];
    if (sqr) {
        sqr_words<6>(z, x.lo);
        sqr_words<6>(z + 12, x.hi);
        sqr_words<6>(z + 24, x.sum);
    } else {
        mul_words<6>(z, x.lo, y.lo);
        mul_words<6>(z + 12, x.hi, y.hi);
        mul_words<6>(z + 24, x.sum, y.sum);
    }
    for (int k = 0; k < kTmCols / 2; k++) {
        uint64_t c[2] = {0, 0};
        for (int h = 0; h < 2; h++)
            for (int i = 0; i < kTmRows; i++)
                c[h] += (uint64_t)((z[i / 4] >> (8 * (i & 3))) & 255u) *
                        im.b[(i / 16 * kTmCols + 2 * k + h) * 16 + i % 16];
        const uint64_t v = c[0] + (c[1] << 8);
        if (v > largest) largest = v;
        w[k] = (uint32_t)v;
    }
    tm_join(r, w);
}
uint64_t shim_tm_largest() { return largest; } // of the joined column pairs: fits 32 bits
}
