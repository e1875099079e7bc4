/* Exhaustive check of the coarse levels' division by the diagonal count
 * (flub_gb300/csrc/coarse.cuh, coarse_half): with y = RN(-1/d), q0 = a y and
 * -q = q0 + (a + d q0) y, the result must equal IEEE a / d for d = 1..6 and
 * every finite float32 a >= 0 (the sequence is odd in a), bit for bit up to
 * the sign of zero.  The one exception: d = 6 and a quotient exactly half-way
 * between two denormals, where it may be the other one of the two.  d = 1, 2
 * and 4 have an exact y and are checked on every 61st value.  Exits 1 on any
 * other mismatch. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

int main(void) {
    long long bad = 0, ties = 0, checked = 0;
    for (int d = 1; d <= 6; d++) {
        const float df = (float)d, y = -1.0f / df;
        const int64_t step = (d & (d - 1)) == 0 ? 61 : 1;
#pragma omp parallel for reduction(+ : bad, ties, checked) schedule(static)
        for (int64_t b = 0; b < 0x7f800000LL; b += step) {
            const uint32_t bits = (uint32_t)b;
            float a;
            memcpy(&a, &bits, 4);
            const float q0 = a * y;
            const float nq = fmaf(fmaf(q0, df, a), y, q0);
            const float q = 0.0f - nq, ref = a / df;
            checked++;
            if (q != ref) {
                const double exact = (double)a / 6.0;
                const int tie = d == 6 && a < 6.0f * 0x1p-126f && fabs((double)q - exact) == 0x1p-150 &&
                                fabs((double)ref - exact) == 0x1p-150;
                ties += tie;
                bad += !tie;
            }
        }
    }
    printf("checked %lld, denormal ties %lld, mismatches %lld\n", checked, ties, bad);
    return bad != 0;
}
