// Test-only host build: element matrices of triangles in the FS_FP64 fixed point
// (csrc/fs_elem_fixed.cuh) and in double (csrc/fs_elem_math.cuh), less the same in
// long double (wide_elem_math.h, the latter header with every double widened).
// Not part of the product.
#include <stdint.h>
#include <string.h>

#include <algorithm>

#include "fs_host_prep.h"
#include "fs_elem_fixed.cuh"
#include "wide_elem_math.h"

using namespace fs;

template <class E> static E element(const double *X, const double *nrm, double t)
{
    E in;
    memset(&in, 0, sizeof in);
    for (int a = 0; a < 3; a++) {
        for (int c = 0; c < 3; c++) {
            in.X[a][c] = X[3 * a + c];
            in.nrm[a][c] = nrm[3 * a + c];
        }
        in.valid[a] = true;
    }
    in.t = t;
    return in;
}

extern "C" {

// n triangles: X, nrm (3 x 3 each), t; of each, 18 x 18: the long double matrix
// (rounded), the fixed point's and the double's difference from it; whether it is
// left to the double kernel
int stretched_triangles(int64_t n, const double *X, const double *nrm, const double *t, const fs_shell_params *p,
                        double *K, double *dfixed, double *ddouble, uint8_t *elongated)
{
    MatConst mc;
    if (prepare_matconst(*p, mc)) return 1;
    fsl::MatConst ml;
    memset(&ml, 0, sizeof ml);
    for (int i = 0; i < 6; i++) ml.Lps[i] = mc.Lps[i];
    for (int i = 0; i < 3; i++) ml.Lt[i] = mc.Lt[i];
    ml.stab_c = mc.stab_c;
    ml.drill_scale = mc.drill_scale;
    typedef CompactRows<3, 2> L;
    static FxSlot mem[(L::SIZE + 1) * FX_GROUP];
    const FxSlots slot{mem};
    for (int64_t e = 0; e < n; e++) {
        const ElemIn<3> in = element<ElemIn<3>>(X + 9 * e, nrm + 9 * e, t[e]);
        const fsl::ElemIn<3> il = element<fsl::ElemIn<3>>(X + 9 * e, nrm + 9 * e, t[e]);
        double rows[11 * 18], F[18][18];
        long double wide[11 * 18];
        t3_rows<double, false, false>(in, mc, nullptr, rows, 18);
        fsl::t3_rows<long double, false, false>(il, ml, nullptr, wide, 18);
        FxGeom<3> geo;
        FxMax mx;
        elongated[e] = t3_coefs(in, mc, slot, geo, mx);
        if (!mx.usable()) return 2;
        const FxExp ex = fx_exponents(mx, 0);
        t3_expand(slot, geo, in.valid, ex);
        for (int p = 0; p < 3; p++)
            for (int q = 0; q < 3; q++) {
                double o[3][6], b[3][6];
                if (p == q) {
                    fx_block_top<1, L::MS, L::BS, L::BSS, true>(slot, 0, p, q, ex, o);
                    fx_block_bottom<1, L::BS, L::BSS, true>(slot, 0, p, q, slot + (L::DR + 3 * p), ex, b);
                    for (int i = 0; i < 3; i++)
                        for (int j = 0; j < 3; j++) b[i][j] = o[j][3 + i];
                } else {
                    fx_block_top<1, L::MS, L::BS, L::BSS, false>(slot, 0, p, q, ex, o);
                    fx_block_bottom<1, L::BS, L::BSS, false>(slot, 0, p, q, slot, ex, b);
                }
                for (int i = 0; i < 3; i++)
                    for (int j = 0; j < 6; j++) {
                        F[6 * p + i][6 * q + j] = o[i][j];
                        F[6 * p + 3 + i][6 * q + j] = b[i][j];
                    }
            }
        for (int i = 0; i < 18; i++)
            for (int j = 0; j < 18; j++) {
                double d = 0;
                long double s = 0;
                for (int r = 0; r < 11; r++) {
                    d = fma(rows[18 * r + i], rows[18 * r + j], d);
                    s += wide[18 * r + i] * wide[18 * r + j];
                }
                const int64_t at = 324 * e + 18 * i + j;
                K[at] = (double)s;
                dfixed[at] = (double)(F[i][j] - s);
                ddouble[at] = (double)(d - s);
            }
    }
    return 0;
}

}  // extern "C"
