// bm_quotient (csrc/fs_beam_math.cuh) against the division, for tests.
#include <stdint.h>

#include "fs_beam_math.cuh"

extern "C" int64_t qc_different(int64_t n, const double *a, const double *b)
{
    int64_t bad = 0;
    for (int64_t i = 0; i < n; i++) bad += fs::bm_quotient(a[i], b[i], 1.0 / b[i]) != a[i] / b[i];
    return bad;
}
