// Test-only host build of the FS_FP64 elements' fixed point
// (csrc/fs_elem_fixed.cuh), beside the same elements in double
// (csrc/fs_elem_math.cuh).  Not part of the product.
#include <stdint.h>
#include <string.h>

#include <algorithm>

#include "fs_host_prep.h"
#include "fs_elem_fixed.cuh"

using namespace fs;

template <int NP, int NN, int MS, int BS, int BSS>
static void blocks(FxSlots rows, int step, int dr, const FxExp &ex, double *K)
{
    for (int p = 0; p < NN; p++)
        for (int q = 0; q < NN; q++) {
            double o[3][6], b[3][6];
            if (p == q) {
                fx_block_top<NP, MS, BS, BSS, true>(rows, step, p, q, ex, o);
                fx_block_bottom<NP, BS, BSS, true>(rows, step, p, q, rows + (dr + 3 * p), ex, b);
                for (int i = 0; i < 3; i++)
                    for (int j = 0; j < 3; j++) b[i][j] = o[j][3 + i];
            } else {
                fx_block_top<NP, MS, BS, BSS, false>(rows, step, p, q, ex, o);
                fx_block_bottom<NP, BS, BSS, false>(rows, step, p, q, rows, ex, b);
            }
            for (int i = 0; i < 3; i++)
                for (int j = 0; j < 6; j++) {
                    K[(6 * p + i) * 6 * NN + 6 * q + j] = o[i][j];
                    K[(6 * p + 3 + i) * 6 * NN + 6 * q + j] = b[i][j];
                }
        }
}

template <int NN> static ElemIn<NN> element(const double *X, const double *nrm, const uint8_t *valid, double t)
{
    ElemIn<NN> in;
    for (int a = 0; a < NN; a++) {
        for (int c = 0; c < 3; c++) {
            in.X[a][c] = X[3 * a + c];
            in.nrm[a][c] = nrm[3 * a + c];
            in.nrmf[a][c] = (float)in.nrm[a][c];
        }
        in.valid[a] = valid[a] != 0;
    }
    in.t = t;
    in.group = 0;
    return in;
}

static void gram(const double *rows, int nrows, int nd, double *K)
{
    for (int i = 0; i < nd; i++)
        for (int j = 0; j < nd; j++) {
            double s = 0.0;
            for (int r = 0; r < nrows; r++) s += rows[r * nd + i] * rows[r * nd + j];
            K[i * nd + j] = s;
        }
}

extern "C" {

// n elements of nen nodes: X, nrm (nen x 3 each), valid (nen), t; fixed and dbl:
// (6 nen)^2 each; usable: whether the fixed point takes the element
int fixed_elements(int nen, int64_t n, const double *X, const double *nrm, const uint8_t *valid, const double *t,
                   const fs_shell_params *p, double *fixed, double *dbl, uint8_t *usable)
{
    MatConst mc;
    if (prepare_matconst(*p, mc)) return 1;
    for (int64_t e = 0; e < n; e++) {
        FxMax mx;
        if (nen == 3) {
            typedef CompactRows<3, 2> L;
            const ElemIn<3> in = element<3>(X + 9 * e, nrm + 9 * e, valid + 3 * e, t[e]);
            static FxSlot mem[(L::SIZE + 1) * FX_GROUP];
            const FxSlots slot{mem};
            FxGeom<3> geo;
            t3_coefs(in, mc, slot, geo, mx);
            usable[e] = mx.usable();
            if (usable[e]) {
                const FxExp ex = fx_exponents(mx, 0);
                t3_expand(slot, geo, in.valid, ex);
                blocks<1, 3, L::MS, L::BS, L::BSS>(slot, 0, L::DR, ex, fixed + 324 * e);
            }
            double rows[11 * 18];
            t3_rows<double, false, false>(in, mc, nullptr, rows, 18);
            gram(rows, 11, 18, dbl + 324 * e);
        } else {
            typedef Q4Compact L;
            const ElemIn<4> in = element<4>(X + 12 * e, nrm + 12 * e, valid + 4 * e, t[e]);
            static FxSlot mem[(L::SIZE + 1) * FX_GROUP];
            const FxSlots slot{mem};
            FxGeom<4> geo[4];
            Q4Elem qe;
            q4_prepare(in, in.t, mc.stab_c, qe);
            double rn[4], tr[4] = {0, 0, 0, 0}, tp[4], td[4] = {0, 0, 0, 0}, rows[36 * 24];
            bool bad = false;
            for (int k = 0; k < 4; k++) {
                const double nn = dot3(in.nrm[k], in.nrm[k]);
                rn[k] = nn > 0.0 ? 1.0 / sqrt(nn) : 0.0;
            }
            for (int j = 0; j < 4; j++) {
                bad |= q4_coefs(qe.Xr, in.nrm, in.valid, rn, in.t, sqrt(qe.stab), j, mc, slot + j * L::GP, geo[j], mx, tp);
                for (int k = 0; k < 4; k++) tr[k] += tp[k];
                q4_point_rows<double, false>(in, qe, j, mc, nullptr, rows + j * 8 * 24, 24, tp);
                for (int k = 0; k < 4; k++) td[k] += tp[k];
            }
            q4_drill_rows<double>(in, td, mc.drill_scale, rows + 32 * 24, 24);
            gram(rows, 36, 24, dbl + 576 * e);
            double sum = 0.0;
            int cnt = 0;
            for (int k = 0; k < 4; k++)
                if (in.valid[k] && rn[k] != 0.0) {
                    sum += tr[k] > 0.0 ? tr[k] / 2 : 0.0;
                    cnt++;
                }
            const double sk = sqrt((cnt ? sum / cnt : 0.0) * mc.drill_scale);
            double dr[4][3];
            for (int k = 0; k < 4; k++)
                for (int c = 0; c < 3; c++) {
                    dr[k][c] = in.valid[k] && rn[k] != 0.0 ? sk * in.nrm[k][c] : 0.0;
                    fx_max(mx.r, dr[k][c]);
                }
            usable[e] = !bad && mx.usable();
            if (!usable[e]) continue;
            const FxExp ex = fx_exponents(mx, 1);
            for (int j = 0; j < 4; j++) {
                fx ax[4][3][3];
                expand_slots<4, L::MS, L::BS, L::BSS>(slot + j * L::GP, geo[j], ex, ax);
            }
            for (int k = 0; k < 4; k++)
                for (int c = 0; c < 3; c++) slot[L::DR + 3 * k + c].x = fx_make(dr[k][c], ex.r);
            blocks<4, 4, L::MS, L::BS, L::BSS>(slot, L::GP, L::DR, ex, fixed + 576 * e);
        }
    }
    return 0;
}

// n doubles x in a group of exponent E: through the limbs and back (a product with one)
void fixed_round_trip(int64_t n, const double *x, int E, double *out)
{
    const fx one = fx_make(1.0, 0);
    for (int64_t i = 0; i < n; i++) out[i] = fx_double(fx_mul(fx_make(x[i], E), one), E);
}

// n dot products of length m of a (exponent ea) and b (exponent eb)
void fixed_dots(int64_t n, int m, const double *a, const double *b, int ea, int eb, double *out)
{
    for (int64_t i = 0; i < n; i++) {
        FxSum s{0, 0};
        for (int k = 0; k < m; k++) fx_mac(s, fx_make(a[i * m + k], ea), fx_make(b[i * m + k], eb));
        out[i] = fx_double(s, ea + eb);
    }
}

}  // extern "C"
